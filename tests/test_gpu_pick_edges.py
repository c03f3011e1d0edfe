"""Peak picking where its sort changes: powers of two of the bitonic sort, the QALEN
cut, the most peaks that are sorted without a threshold, the largest spectrum sorted in shared memory and the ones past it, with
distinct intensities, a few equal ones (among the kept peaks, across the cut, below
it) and only equal ones; against the reader's restatement."""
import numpy as np
import pytest

from oracle import ms2 as M
from tests.test_gpu_ms2 import _device_batch, _index, _same

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 2, 3, 31, 32, 33, 99, 100, 101, 102, 127, 128, 129, 512, 513, 1024, 1025, 1500]


@pytest.mark.parametrize("kind", ["distinct", "few", "cut", "below", "levels", "steps", "all", "zero"])
@pytest.mark.parametrize("pick", [(100, 100000, 1000), (10, 5000, 0)])
def test_pick_at_sort_edges(kind, pick, tmp_path):
    rng = np.random.default_rng(17)
    lines = ["H\tx\n"]
    for s, n in enumerate(SIZES):
        lines.append(f"S\t{s}\t{s}\t500\nZ\t2\t{1000 + s}.5\nI\tRTime\t{s}.25\n")
        it = rng.permutation(np.arange(1, n + 1)) * 1.25 + 100.0
        o = np.argsort(it)[::-1]
        if kind == "few" and n > 9:
            it[o[5:8]] = it[o[5]]
        if kind == "cut" and n > 101:
            it[o[98:102]] = it[o[98]]
        if kind == "below" and n > 128:
            it[o[110:120]] = it[o[110]]
        if kind == "levels":  # groups of equal ones everywhere
            it = np.floor(it / (100 if n > 200 else 12))
        if kind == "steps":  # ... in ascending order, the largest group across the cut
            it = np.sort(np.floor(it / 40))
        if kind == "all":
            it[:] = 77.5
        if kind == "zero":
            it[:] = 0.0
        mz = rng.uniform(100, 2000, n)
        lines += [f"{a:.4f} {b:.2f}\n" for a, b in zip(mz, it)]
    path = tmp_path / "e.ms2"
    path.write_text("".join(lines))
    st, o = M.read_ms2(str(path), *pick)
    assert st == 0
    ix = _index(*pick)
    _same(_device_batch(ix, str(path)), o)
    _same(_device_batch(ix, str(path), 4), o)
    ix.close()
