"""What the library keeps of freed device memory can be given back, and calls
after that work as before."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_freed_memory_goes_back(wct, synth):
    import torch
    rows, cols = 10000, 6000
    x = torch.randn((rows, cols), dtype=torch.complex64, device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    # modules, streams and plans are loaded and made by first calls, and stay
    wct.dft_2d_device(x.data_ptr(), y.data_ptr(), rows, cols)
    wct.from_config(synth.plane1_config(nticks=2000))(synth.plane1_depos(n=500, seed=1))
    torch.cuda.synchronize()
    wct.release_memory()
    before = free()
    wct.dft_2d_device(x.data_ptr(), y.data_ptr(), rows, cols)
    kept = free()
    dt = wct.from_config(synth.plane1_config(nticks=2000))
    depos = synth.plane1_depos(n=500, seed=1)
    first, _, _ = dt(depos)
    wct.release_memory()
    second, _, _ = dt(depos)
    assert np.array_equal(first, second)
    del dt
    wct.release_memory()
    after = free()
    # one transposed copy of 480 MB; what tables of live plans hold of a mapped piece (32 MiB each) stays
    scratch, piece = 8 * rows * cols, 32 << 20
    assert before - kept >= scratch - 2 * piece
    assert before - after <= 2 * piece
    wct.dft_2d_device(x.data_ptr(), z.data_ptr(), rows, cols)
    torch.cuda.synchronize()
    assert torch.equal(y, z)
