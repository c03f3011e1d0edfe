"""Files large enough for the device's parser: every form of line it takes itself,
lines across its 8 KB tiles, and the forms it leaves to the host's parser; the batch
equals the restated reader's and the raw peaks the host parser's."""
import numpy as np
import pytest

from oracle import ms2 as M
from tests.test_gpu_ms2 import _device_batch, _index, _same

pytestmark = pytest.mark.gpu


def _body(rng, nspec, eol, fmt):
    out = []
    for s in range(nspec):
        out.append(f"S\t{s}\t{s}\t{500 + s}.5{eol}")
        if s % 3:
            out.append(f"I\tRTime\t{s}.125{eol}")
            out.append(f"I\tOther\t{s}{eol}")
        if s % 4:
            out.append(f"Z\t{s % 5}\t{1000 + s}.0625{eol}")
        n = int(rng.integers(0, 400))
        mz, it = rng.uniform(100, 2000, n), rng.lognormal(6, 2, n)
        out += [fmt(i, a, b) + eol for i, (a, b) in enumerate(zip(mz, it))]
    return out


FORMS = {
    "plain": lambda i, a, b: f"{a:.4f} {b:.1f}",
    "wide": lambda i, a, b: ("  " * (i % 3)) + f"{a:.11f}{' ' * (1 + i % 4)}{b:.8f}",
    "tokens": lambda i, a, b: f"{int(a)} {b:.2f} 3 x" if i % 2 else f"{a:.3f} {int(b)}. ",
}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("eol", ["\n", "\r\n"])
def test_device_parse_equals_reader(form, eol, tmp_path):
    from hicops_gb300 import dslim
    rng = np.random.default_rng(len(form) + len(eol))
    lines = [f"H\t{'x' * 9000}{eol}", f"D\tnote{eol}", f"150.5 20.25{eol}", f"Z\t3\t777.5{eol}"]  # before the first S
    lines += _body(rng, 400, eol, FORMS[form])
    text = "".join(lines)[:-len(eol)]  # no newline at the end
    assert len(text) > 1 << 20
    path = str(tmp_path / "d.ms2")
    open(path, "wb").write(text.encode())
    pick = (100, 100000, 1000)
    st, o = M.read_ms2(path, *pick)
    assert st == 0
    ix = _index(*pick)
    _same(_device_batch(ix, path), o)
    _same(_device_batch(ix, path, 100), o)
    raw = dslim.read_ms2_raw(path, 100)  # the host's parser
    import ctypes as C
    from hicops_gb300 import _lib as L
    r = dslim.MSQuery(ix).initialize(path)
    assert (r.QAcount, r.maxslen) == (raw["prec"].size, raw["maxslen"])
    n = r.QAcount
    off, mz, it = np.zeros(n + 1, np.uint64), np.zeros_like(raw["mz"]), np.zeros_like(raw["mz"])
    assert ix.lib.hc_ms2_raw(r.h, 0, n, L.ptr(off), L.ptr(mz), L.ptr(it), None, None, None) == 0
    assert np.array_equal(off, raw["off"]) and np.array_equal(mz, raw["mz"]) and np.array_equal(it, raw["intensity"])
    r.DeinitQueryFile()
    ix.close()


@pytest.mark.parametrize("odd", ["1e2 5", "+3 4", "100\t5", "100", "\r", "12.5.5 3", "1234567890123456.5 1", "99999999999 1",
                                 "100 5e1", " ", "100 5\x005"])
def test_odd_lines_take_the_host_parser(odd, tmp_path):
    rng = np.random.default_rng(3)
    lines = _body(rng, 400, "\n", FORMS["plain"])
    lines.insert(len(lines) // 2, odd + "\n")
    text = "".join(lines)
    assert len(text) > 1 << 20
    path = str(tmp_path / "o.ms2")
    open(path, "wb").write(text.encode())
    pick = (100, 100000, 1000)
    from hicops_gb300 import dslim
    raw = dslim.read_ms2_raw(path, 100)
    ix = _index(*pick)
    r = dslim.MSQuery(ix).initialize(path)
    from hicops_gb300 import _lib as L
    n = r.QAcount
    off, mz, it = np.zeros(n + 1, np.uint64), np.zeros_like(raw["mz"]), np.zeros_like(raw["mz"])
    assert ix.lib.hc_ms2_raw(r.h, 0, n, L.ptr(off), L.ptr(mz), L.ptr(it), None, None, None) == 0
    assert np.array_equal(off, raw["off"]) and np.array_equal(mz, raw["mz"]) and np.array_equal(it, raw["intensity"])
    r.DeinitQueryFile()
    ix.close()
