"""Entry points called with plain lists of tensors where they take device arrays
of pointers: each list's array lives until the call has launched, on the
current stream and on a stream given to the call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def frame(native):
    import gpu_runner as R
    from cases import Case
    fr = R.Frame(Case(128, 96, seed=71, border_mode=1))
    return fr, R.convert(fr)


@pytest.mark.parametrize("side", [False, True])
def test_lists_of_tensors(frame, side):
    import torch
    from tile_processor_gpu_b200 import api
    fr, want = frame
    c = fr.case
    stream = torch.cuda.Stream() if side else None
    clt = [torch.zeros_like(x) for x in fr.clt]
    torch.cuda.synchronize()
    if side:
        # the call waits behind this while the caller goes on allocating
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)
    api.convert_correct_tiles(fr.g, fr.extra, fr.kernels, fr.images, fr.tasks, clt, c.dstride, c.num_tiles, 0,
                              stream=stream)
    later = [torch.zeros(4, dtype=torch.int64, device="cuda") for _ in range(64)]
    torch.cuda.synchronize()
    del later
    assert all(np.array_equal(a.cpu().numpy(), b) for a, b in zip(clt, want))
