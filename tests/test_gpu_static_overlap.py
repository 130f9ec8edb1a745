"""bh_sort_keys_static with outputs that overlap the inputs: every sort reads all its inputs before it writes
an output, in two launches (up to 32 768 keys) and in three."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 37, 128, 4096])
@pytest.mark.parametrize("n", [1000, 32768, 32769, 40001, 65536])
def test_overlapping_outputs(bh, n, shift):
    torch = pytest.importorskip("torch")
    lib = bh.load()
    rng = np.random.default_rng(n + shift)
    keys = rng.integers(0, 1 << 16, n).astype(np.int64)  # ties
    kbuf = torch.zeros(n + shift, dtype=torch.int64, device="cuda")
    vbuf = torch.zeros(n + shift, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    order = np.argsort(keys, kind="stable")
    for up in (True, False):  # the outputs `shift` elements below or above the inputs
        i, o = (shift, 0) if up else (0, shift)
        kbuf[i : i + n] = torch.from_numpy(keys)
        vbuf[i : i + n] = torch.arange(n, dtype=torch.int32)
        rc = lib.bh_sort_keys_static(kbuf.data_ptr() + 8 * i, vbuf.data_ptr() + 4 * i, kbuf.data_ptr() + 8 * o,
                                     vbuf.data_ptr() + 4 * o, n, stream, None)
        torch.cuda.synchronize()
        assert rc == 0
        assert np.array_equal(kbuf[o : o + n].cpu().numpy(), keys[order])
        assert np.array_equal(vbuf[o : o + n].cpu().numpy(), order)
