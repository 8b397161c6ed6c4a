"""GPU tests of the per-vertex SH kernel's staging forms, bit for bit against the oracle: odd
coefficient counts (one bulk copy), multiples of 4 (rows of 16-byte chunks, with and without
padding), the other even ones, and transfer matrices that start on no 16-byte boundary."""
import numpy as np
import pytest

from neural_wavelet_prt_demo_b200 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 8, 16, 25, 31, 32, 33, 36, 49, 62, 64, 65, 72, 80, 81])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_sh_vertex_forms_bit_exact(cuda, n, shift):
    import torch
    from neural_wavelet_prt_demo_b200 import engine as eng
    V = 19
    T, brdf, _, _ = synth.make_sh_mesh(V, 1, 81, seed=n)
    T, brdf = T[:, :n, :n].copy(), brdf[:, :n].copy()
    L = synth.make_sh_transport(3, 81, seed=5).T[:n].copy()
    buf = torch.empty(T.size + shift, dtype=torch.float32, device=cuda)
    Td = buf[shift:].view(V, n, n)
    Td.copy_(torch.from_numpy(T))
    got = eng.sh_vertex_radiance(Td, *(torch.from_numpy(a).to(cuda) for a in (brdf, L))).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), O.sh_vertex_radiance(T, brdf, L).view(np.uint32))


@pytest.mark.parametrize("n", [1, 9, 33, 36, 62, 64, 81])
def test_sh_vertex_waits_that_run_out_lose_nothing(cuda, n):
    # the call has no status for a wait that gave up, so the results have to be right all the same
    import torch
    from neural_wavelet_prt_demo_b200 import _lib
    V = 2501  # more than the blocks' warps: a warp goes on after the wait that ran out
    T, brdf, _, _ = synth.make_sh_mesh(V, 1, 81, seed=n)
    T, brdf = T[:, :n, :n].copy(), brdf[:, :n].copy()
    L = synth.make_sh_transport(3, 81, seed=5).T[:n].copy()
    Td, bd, Ld = (torch.from_numpy(a).to(cuda) for a in (T, brdf, L))
    out = torch.full((V, 3), float("nan"), device=cuda)
    _lib.check(_lib.lib().nwprt_selftest_sh_vertex(Td.data_ptr(), bd.data_ptr(), Ld.data_ptr(), V, n, out.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream))
    assert np.array_equal(out.cpu().numpy().view(np.uint32), O.sh_vertex_radiance(T, brdf, L).view(np.uint32))


@pytest.mark.parametrize("n", [10, 24, 44, 48, 56, 78])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_sh_vertex_even_rows_bit_exact(cuda, n, shift):
    import torch
    from neural_wavelet_prt_demo_b200 import engine as eng
    V = 1300  # several per warp
    T, brdf, _, _ = synth.make_sh_mesh(V, 1, 81, seed=n)
    T, brdf = T[:, :n, :n].copy(), brdf[:, :n].copy()
    L = synth.make_sh_transport(3, 81, seed=5).T[:n].copy()
    buf = torch.empty(T.size + shift, dtype=torch.float32, device=cuda)
    Td = buf[shift:].view(V, n, n)
    Td.copy_(torch.from_numpy(T))
    got = eng.sh_vertex_radiance(Td, *(torch.from_numpy(a).to(cuda) for a in (brdf, L))).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), O.sh_vertex_radiance(T, brdf, L).view(np.uint32))


@pytest.mark.parametrize("n,shift", [(62, 0), (72, 1)])
def test_sh_vertex_even_counts_keep_up_with_odd_ones(cuda, n, shift):
    # 4-byte copies to an odd stride took 3.1 and 2.8 times as long as the next smaller, odd count
    import torch
    from neural_wavelet_prt_demo_b200 import engine as eng

    def us(m):
        V = 15_000_000 // (m * m)
        T = torch.randn(V * m * m + shift, device=cuda)[shift:].view(V, m, m)
        brdf, L = torch.randn((V, m, 3), device=cuda), torch.randn((m, 3), device=cuda)
        times = []
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(20):
                eng.sh_vertex_radiance(T, brdf, L)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return sorted(times[2:])[3]

    assert us(n) < 2.2 * us(n - 1)
