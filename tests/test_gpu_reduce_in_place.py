"""The sizes from which sppm_reduce_texture's later launches fold the scratch in place (one level at 4096,
two at 8192, four through shared memory at 16384), against the fold written level by level in torch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fold(t, op, torch):
    """min.fs / max.fs / sum.fs of the four quadrants' texels, down to one."""
    while t.shape[0] > 1:
        n = t.shape[0] // 2
        a, b, c, d = t[:n, :n], t[:n, n:], t[n:, :n], t[n:, n:]
        if op == 2:
            t = ((a + b) + c) + d
        else:
            f = torch.fmin if op == 0 else torch.fmax
            t = f(f(a, b), f(c, d))
    return t[0, 0].cpu().numpy()


@pytest.mark.parametrize("R", [4096, 8192, 16384])
def test_in_place_levels(R):
    torch = pytest.importorskip("torch")
    import glslppm_gb300 as g
    t = torch.randn((R, R, 4), generator=torch.Generator("cuda").manual_seed(R), device="cuda") * 100
    for op in (0, 1, 2):
        got = g.renderer.reduce_texture(t.data_ptr(), R, op, torch.cuda.current_stream().cuda_stream)
        np.testing.assert_array_equal(got.view(np.uint32), fold(t, op, torch).view(np.uint32), err_msg=f"{R} op {op}")
