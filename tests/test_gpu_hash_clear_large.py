"""sppm_hash_build clears tables of nearly 2^32 slots, and nothing past their end: four slots a thread, where
the index of the last thread's four plus four is 2^32."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("below", [512, 1021, 2048])
def test_a_table_of_nearly_two_to_the_32(below):
    torch = pytest.importorskip("torch")
    from glslppm_gb300 import renderer
    total, step = 1 << 32, 1 << 29
    n = total - below
    if torch.cuda.mem_get_info()[0] < 48 << 30:
        pytest.skip("needs two tables of 16 GiB")
    winner = torch.full((total,), 7, dtype=torch.int32, device="cuda")
    count = torch.full((total,), 7, dtype=torch.int32, device="cuda")
    pos, flux = torch.zeros((16, 4), device="cuda"), torch.full((16, 4), -1.0, device="cuda")  # no photon is stored
    renderer.hash_build(pos.data_ptr(), flux.data_ptr(), 4, 4, n, (0.0, 0.0, 0.0), 1.0, 0, winner.data_ptr(),
                        count.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for table, empty in ((winner, -1), (count, 0)):
        for i in range(0, n, step):
            part = table[i:min(i + step, n)]
            assert int(part.min()) == int(part.max()) == empty, i
        assert bool((table[n:] == 7).all())


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 1023, 1024, 1025])
def test_small_tables(n, offset):
    torch = pytest.importorskip("torch")
    from glslppm_gb300 import renderer
    winner = torch.full((n + 16,), 7, dtype=torch.int32, device="cuda")
    count = torch.full((n + 16,), 7, dtype=torch.int32, device="cuda")
    pos, flux = torch.zeros((16, 4), device="cuda"), torch.full((16, 4), -1.0, device="cuda")
    renderer.hash_build(pos.data_ptr(), flux.data_ptr(), 4, 4, n, (0.0, 0.0, 0.0), 1.0, 0,
                        winner.data_ptr() + 4 * offset, count.data_ptr() + 4 * offset,
                        torch.cuda.current_stream().cuda_stream)
    for table, empty in ((winner, -1), (count, 0)):
        want = torch.full((n + 16,), 7, dtype=torch.int32, device="cuda")
        want[offset:offset + n] = empty
        assert torch.equal(table, want)
