"""The CTA pairs of the 4-bit tensor GEMM under many repetitions: every call's
recovery words equal the table kernel's, bit for bit.  A stage that a pair's
MMAs read before the other CTA's part of it is in place shows up as a wrong
word now and then, so the calls have several tiles per pair and are repeated
without a wait between them."""
import pytest

from parpar_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R,words,reps", [
    (10, 2, 128 * 2048, 60),     # whole passes in one stage, several passes to an accumulator group
    (60, 40, 128 * 1024, 60),    # one stage a pass, one column tile
    (100, 10, 128 * 2048, 60),   # full stages, narrow tiles
    (777, 133, 128 * 700, 20),   # several stages a pass, three column tiles
    (2000, 200, 128 * 460, 20),  # single-bit passes over one full column tile
    (1920, 480, 128 * 380, 10),  # single-bit passes, two column tiles
])
def test_pairs_agree_with_the_table_kernel_every_time(n, R, words, reps):
    import torch
    L = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(n)
    d_in, d_coeff = (torch.randint(-32768, 32768, shape, generator=g, device="cuda").to(torch.int16)
                     for shape in ((n, words), (R, n)))
    st = torch.cuda.current_stream().cuda_stream

    def call(rec, method, sb):
        scratch = torch.empty(sb, dtype=torch.uint8, device="cuda")
        assert L.par2cuda_muladd(d_in.data_ptr(), words, n, d_coeff.data_ptr(), rec.data_ptr(), words, R, words, 0, method,
                                 scratch.data_ptr(), sb, st) == 0, L.par2cuda_last_error()

    want = torch.empty((R, words), dtype=torch.int16, device="cuda")
    call(want, _lib.METHOD_COMB, L.par2cuda_muladd_scratch_bytes(R, n))
    sb = L.par2cuda_tensor_fp4_scratch_bytes(R, n, words)
    got = [torch.empty_like(want) for _ in range(2)]
    wrong = torch.zeros((), dtype=torch.int64, device="cuda")
    for k in range(reps):
        rec = got[k & 1]
        rec.zero_()
        call(rec, _lib.METHOD_TENSOR_FP4, sb)
        wrong += (rec != want).sum()
    assert int(wrong) == 0
    assert L.par2cuda_device_error() == 0
