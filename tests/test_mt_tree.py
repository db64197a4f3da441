"""The device MT19937 stream's tree of jumps (k_mt_seed, k_mt_jump) at the
edges of its segments: one word, a window, a segment and one word more, odd
segment counts, a last segment shorter than a window, and counts whose levels
split a jump over several CTAs.  Words equal NumPy's MT19937 of the same seed
(init_genrand) exactly."""
import numpy as np
import pytest

from rrtmg_sw_gb300 import interface as gi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_seg,n", [(10, 1), (10, 623), (10, 1024), (10, 1025), (10, 3 * 1024 + 7),
                                       (10, 33 * 1024 + 623), (15, (1 << 15) + 1), (15, 5 * (1 << 15) + 625),
                                       (12, 331 * 4096 + 1), (0, 1), (0, 100_003)])
def test_stream_words(log_seg, n):
    torch = pytest.importorskip("torch")
    from rrtmg_sw_gb300 import build
    build.build()
    gi.rrtmg_sw_ini(1.004e3)
    out = torch.full((n + 8,), -1, dtype=torch.int32, device="cuda")
    gi.mt_stream_dev(20261, n, out.data_ptr(), log_seg, torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    g = np.random.MT19937()
    g._legacy_seeding(20261)
    np.testing.assert_array_equal(got[:n].view(np.uint32), g.random_raw(n).astype(np.uint32))
    assert np.all(got[n:] == -1)  # nothing past the stream
