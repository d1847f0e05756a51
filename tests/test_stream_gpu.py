"""Stream compaction and scan at the edges of their slices, phases and count rows."""
import numpy as np
import pytest

from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu

SLICE = 32 * 1024  # bytes of a compaction slice; a phase is one slice on each of 152 SMs
EDGES = [0, 1, 2, 151, 152, 153, 2 * 152, 3 * 152 - 1, 7 * 152 + 1, 8 * 152, 9 * 152 + 75]


@pytest.mark.parametrize("elem", [4, 8, 16])
@pytest.mark.parametrize("slices", EDGES)
def test_compaction_at_phase_edges(hx, slices, elem):
    """Exactly the scratch that is asked for, guarded behind; every selected share from none to all."""
    for off in (-1, 0, 1):
        n = slices * (SLICE // elem) + off
        if n < 1:
            continue
        rng = np.random.default_rng(n)
        words = rng.integers(0, 100, size=(n, elem // 4), dtype=np.uint32)
        if elem == 16:
            words[:, 1] = words[:, 3] = 0
        x = to_dev(words)
        out = to_dev(np.full_like(words, 7))
        need = hx.tools.scratch_bytes(hx.SCRATCH_COPY_IF, n)
        guard = to_dev(np.full(need + 256, 0xA5, np.uint8))
        for share in (0, 1, 50, 100):
            pred = hx.Pred.mod_lt(100, share) if elem == 4 else hx.Pred(hx.PRED_MOD_LT, hx.FIELD_VALUE, 100, share)
            value = words[:, 0] if elem == 4 else words[:, elem // 8]
            want = words[value % 100 < share]
            c = hx.tools.copy_if(x, out, pred, elem_bytes=elem, scratch=guard, scratch_bytes=need)
            assert c == len(want)
            np.testing.assert_array_equal(from_dev(out, np.uint32).reshape(n, -1)[:c], want)
        assert (from_dev(guard, np.uint8)[need:] == 0xA5).all()


@pytest.mark.parametrize("slices", EDGES)
def test_scan_at_phase_edges(hx, slices):
    for off in (-1, 0, 1):
        n = slices * 16384 + off
        if n < 1:
            continue
        x = np.random.default_rng(n).integers(0, 1 << 32, size=n, dtype=np.uint32)
        out = to_dev(np.zeros(n, np.uint32))
        hx.tools.split_prefix_scan(to_dev(x), out)
        want = np.zeros(n, np.uint32)
        np.cumsum(x[:-1], dtype=np.uint32, out=want[1:])
        np.testing.assert_array_equal(from_dev(out, np.uint32), want)
