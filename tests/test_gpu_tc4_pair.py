"""The CTA pairs of the 4-bit tensor GEMM under many repetitions: every call's
recovery words equal the table kernel's, bit for bit.  A stage that a pair's
MMAs read before the other CTA's part of it is in place shows up as a wrong
word now and then, so the calls have several tiles per pair and are repeated
without a wait between them."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from parpar_gb300 import _lib

pytestmark = pytest.mark.gpu


def plan_of(L, n, R, words):
    plan = _lib.Fp4Plan()
    sb = L.par2cuda_tensor_fp4_scratch_bytes(R, n, words)
    assert L.par2cuda_tensor_fp4_plan(R, n, words, sb, 0, ctypes.byref(plan)) == 0, L.par2cuda_last_error()
    return plan


def form_of(L, n, R, words):
    return plan_of(L, n, R, words).form


@pytest.mark.parametrize("n,R,words,form,reps", [
    (10, 2, 128 * 2048, 4, 60),     # whole passes in one stage, several passes to an accumulator group
    (60, 40, 128 * 1024, 4, 60),    # one stage a pass, one column tile
    (100, 10, 128 * 2048, 4, 60),   # full stages, narrow tiles
    (777, 133, 128 * 700, 4, 20),   # several stages a pass, three column tiles
    (2000, 200, 128 * 152, 1, 40),  # single-bit passes over one full column tile
    (1920, 480, 128 * 380, 1, 10),  # single-bit passes, two column tiles, several tiles per pair
])
def test_pairs_agree_with_the_table_kernel_every_time(n, R, words, form, reps):
    import torch
    L = _lib.load()
    assert form_of(L, n, R, words) == form
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


@pytest.mark.parametrize("n,R,words", [(960, 240, 19456), (961, 472, 19301), (1437, 240, 38000), (2000, 200, 19455), (4096, 480, 9728)])
def test_long_passes_are_single_bit_passes(n, R, words):
    # the sizes that test_gpu_tensor_fp4.py compares with the table kernel for their sake
    assert form_of(_lib.load(), n, R, words) == 1


def test_single_bit_passes_agree_with_the_field():
    # every coefficient bit against every word bit, at every input's place in a unit of 96
    import torch
    L = _lib.load()
    n, R, words, unit, seg = 960, 240, 19456, 96, 256
    assert form_of(L, n, R, words) == 1
    x = np.zeros((unit, unit // 16 * seg), dtype=np.uint16)
    for i in range(unit):
        at = i // 16 * seg + i % 16 * 16
        x[i, at:at + 16] = 1 << np.arange(16, dtype=np.uint32)
    coeff = np.zeros((R, n), dtype=np.uint16)
    coeff[:, :unit] = [[1 << ((r + i) % 16) for i in range(unit)] for r in range(R)]
    d_in = torch.zeros((n, words), dtype=torch.int16, device="cuda")
    d_in[:unit, :x.shape[1]] = torch.from_numpy(x.view(np.int16)).cuda()
    d_coeff = torch.from_numpy(coeff.view(np.int16)).cuda()
    d_rec = torch.full((R, words), -1, dtype=torch.int16, device="cuda")
    sb = L.par2cuda_tensor_fp4_scratch_bytes(R, n, words)
    scratch = torch.empty(sb, dtype=torch.uint8, device="cuda")
    assert L.par2cuda_muladd(d_in.data_ptr(), words, n, d_coeff.data_ptr(), d_rec.data_ptr(), words, R, words, 0,
                             _lib.METHOD_TENSOR_FP4, scratch.data_ptr(), sb, None) == 0
    torch.cuda.synchronize()
    want = O.recover_coeffs(x.view(np.uint8), np.full(unit, 2 * x.shape[1]), coeff[:, :unit].copy()).view(np.int16)
    got = d_rec.cpu().numpy()
    assert np.array_equal(got[:, :x.shape[1]], want) and not got[:, x.shape[1]:].any()


@pytest.mark.parametrize("n,R,words,splits", [
    (289, 1, 2, 7), (300, 7, 130, 7), (500, 30, 2052, 7),    # one tile and several, a last one of two words
    (1000, 60, 256 * 10, 7), (1000, 61, 256 * 9, 4),         # one column tile and two
    (3000, 33, 256 * 19, 4), (3000, 33, 256 * 19 + 2, 1),    # both sides of the line
    (500, 30, 2051, 1),                                      # an odd number of words
])
@pytest.mark.parametrize("acc", [0, 1])
@pytest.mark.parametrize("off", [0, 1])
def test_split_passes_match_the_table_kernel(n, R, words, splits, acc, off):
    # off: recovery rows off 4-byte boundaries (never split)
    import torch
    L = _lib.load()
    assert plan_of(L, n, R, words).pass_splits == splits
    g = torch.Generator(device="cuda").manual_seed(n + words)
    pw = (words + 63) // 64 * 64
    d_in, start, d_coeff = (torch.randint(-32768, 32768, shape, generator=g, device="cuda").to(torch.int16)
                            for shape in ((n, pw), (R, pw), (R, n)))
    got = {}
    for method in (_lib.METHOD_COMB, _lib.METHOD_TENSOR_FP4):
        at = off if method == _lib.METHOD_TENSOR_FP4 else 0
        buf = torch.full((R * pw + 2,), 0x5A5A, dtype=torch.int16, device="cuda")
        rec = buf[at:at + R * pw].view(R, pw)
        rec.copy_(start)
        sb = L.par2cuda_muladd_scratch_bytes(R, n) if method == _lib.METHOD_COMB else \
            L.par2cuda_tensor_fp4_scratch_bytes(R, n, words)
        scratch = torch.empty(sb, dtype=torch.uint8, device="cuda")
        assert L.par2cuda_muladd(d_in.data_ptr(), pw, n, d_coeff.data_ptr(), rec.data_ptr(), pw, R, words, acc, method,
                                 scratch.data_ptr(), sb, None) == 0, L.par2cuda_last_error()
        torch.cuda.synchronize()
        got[method] = rec
        assert buf[R * pw + at:].eq(0x5A5A).all() and buf[:at].eq(0x5A5A).all()
    assert L.par2cuda_device_error() == 0
    assert torch.equal(got[_lib.METHOD_COMB][:, :words], got[_lib.METHOD_TENSOR_FP4][:, :words])
    # nothing past the words was written
    assert torch.equal(got[_lib.METHOD_TENSOR_FP4][:, words:], start[:, words:])


@pytest.mark.parametrize("acc", [0, 1])
def test_split_passes_in_a_captured_graph(acc):
    import torch
    L = _lib.load()
    n, R, words = 500, 30, 2052
    assert plan_of(L, n, R, words).pass_splits == 7
    g = torch.Generator(device="cuda").manual_seed(3)
    pw = (words + 63) // 64 * 64
    d_in, start, d_coeff = (torch.randint(-32768, 32768, shape, generator=g, device="cuda").to(torch.int16)
                            for shape in ((n, pw), (R, pw), (R, n)))
    rec = start.clone()
    sb = L.par2cuda_tensor_fp4_scratch_bytes(R, n, words)
    scratch = torch.empty(sb, dtype=torch.uint8, device="cuda")

    def call(out):
        assert L.par2cuda_muladd(d_in.data_ptr(), pw, n, d_coeff.data_ptr(), out.data_ptr(), pw, R, words, acc,
                                 _lib.METHOD_TENSOR_FP4, scratch.data_ptr(), sb,
                                 torch.cuda.current_stream().cuda_stream) == 0, L.par2cuda_last_error()

    want = start.clone()
    call(want)                                   # also loads the kernels before the capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(rec)
    for _ in range(3):
        rec.copy_(start)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(rec, want)
    assert L.par2cuda_device_error() == 0
