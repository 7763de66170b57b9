"""GPU hashing (IFSC slice MD5+CRC32, file MD5, packet MD5) vs the golden
vectors recorded from the reference hasher and vs the oracle."""
import hashlib
import json
import os
import zlib

import numpy as np
import pytest

from oracle import oracle as O
from parpar_gb300 import _lib, synth

pytestmark = pytest.mark.gpu
GOLDEN = json.load(open(os.path.join(os.path.dirname(__file__), "golden", "golden.json")))


def _rows_from_files(torch, files, S):
    """Lays files out as consecutive rows of S bytes (row pitch from the library)."""
    L = _lib.load()
    pitch = L.par2cuda_row_pitch_bytes(S)
    nrows = sum((len(f) + S - 1) // S for f in files)
    host = np.zeros((max(nrows, 1), pitch), np.uint8)
    lens, first, r = [], [], 0
    for f in files:
        first.append(r)
        for off in range(0, len(f), S):
            chunk = f[off:off + S]
            host[r, :len(chunk)] = chunk
            lens.append(len(chunk))
            r += 1
    d = torch.from_numpy(host).cuda()
    return d, pitch, np.array(lens, np.uint32), np.array(first, np.uint32), nrows


def _hash(torch, files, S):
    L = _lib.load()
    d, pitch, lens, first, nrows = _rows_from_files(torch, files, S)
    d_lens = torch.from_numpy(lens.view(np.int32)).cuda()
    ifsc = torch.zeros(max(nrows, 1) * 20, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_slice_hash(d.data_ptr(), pitch, nrows, d_lens.data_ptr(), S, ifsc.data_ptr(), None), "slice_hash")
    flen = torch.tensor([len(f) for f in files], dtype=torch.int64, device="cuda")
    d_first = torch.from_numpy(first.view(np.int32)).cuda()
    md5 = torch.zeros(16 * len(files), dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_file_md5(d.data_ptr(), pitch, len(files), flen.data_ptr(), d_first.data_ptr(), S, md5.data_ptr(), None), "file_md5")
    torch.cuda.synchronize()
    return ifsc.cpu().numpy()[: nrows * 20].tobytes(), md5.cpu().numpy().tobytes()


@pytest.mark.parametrize("case", GOLDEN["hash"], ids=lambda c: c["name"])
def test_golden_ifsc_and_file_md5(case):
    torch = pytest.importorskip("torch")
    data = synth.slice_bytes(case["seed"], 0, case["len"])
    ifsc, md5 = _hash(torch, [data], case["slice"])
    assert ifsc.hex() == case["ifsc"]
    assert md5.hex() == case["file_md5"]


def test_many_files_uneven():
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(11)
    S = 4096
    files = [synth.slice_bytes(100 + k, 0, int(l)) for k, l in enumerate(rng.integers(1, 5 * S, size=23))]
    files.append(synth.slice_bytes(999, 0, 3 * S))  # exact multiple
    ifsc, md5 = _hash(torch, files, S)
    exp_ifsc = b"".join(O.hash_file(f, S)[0] for f in files)
    assert ifsc == exp_ifsc
    assert md5 == b"".join(hashlib.md5(f.tobytes()).digest() for f in files)


@pytest.mark.parametrize("S", [4, 8, 60, 64, 68, 1000, 65536 + 4])
def test_slice_sizes_not_block_aligned(S):
    torch = pytest.importorskip("torch")
    files = [synth.slice_bytes(S, 0, 3 * S + S // 2 + 2), synth.slice_bytes(S + 1, 0, 2)]
    ifsc, md5 = _hash(torch, files, S)
    assert ifsc == b"".join(O.hash_file(f, S)[0] for f in files)
    assert md5 == b"".join(hashlib.md5(f.tobytes()).digest() for f in files)
    # each IFSC CRC equals zlib's CRC of the zero-padded slice
    d = files[0]
    blk = d[:S].tobytes()
    assert int.from_bytes(ifsc[16:20], "little") == zlib.crc32(blk)


@pytest.mark.parametrize("case", GOLDEN["md5multi"], ids=lambda c: "n%d_len%d" % (c["n"], c["len"]))
def test_rows_md5_golden(case):
    torch = pytest.importorskip("torch")
    L = _lib.load()
    n, ln = case["n"], case["len"]
    bufs = synth.slices(case["seed"], 0, n, ln)
    pitch = L.par2cuda_row_pitch_bytes(ln)
    host = np.zeros((n, pitch), np.uint8)
    host[:, :ln] = bufs
    d = torch.from_numpy(host).cuda()
    out = torch.zeros(16 * n, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_rows_md5(d.data_ptr(), pitch, n, ln, None, 0, out.data_ptr(), None), "rows_md5")
    torch.cuda.synchronize()
    assert out.cpu().numpy().tobytes().hex() == case["md5"]


def test_rows_md5_with_packet_prefix():
    torch = pytest.importorskip("torch")
    L = _lib.load()
    n, ln, pl = 5, 4100, 36
    bufs = synth.slices(3, 0, n, ln)
    pre = synth.slices(4, 0, n, pl)
    pitch = L.par2cuda_row_pitch_bytes(ln)
    host = np.zeros((n, pitch), np.uint8)
    host[:, :ln] = bufs
    d = torch.from_numpy(host).cuda()
    dp = torch.from_numpy(np.ascontiguousarray(pre)).cuda()
    out = torch.zeros(16 * n, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_rows_md5(d.data_ptr(), pitch, n, ln, dp.data_ptr(), pl, out.data_ptr(), None), "rows_md5")
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(n, 16)
    for i in range(n):
        assert got[i].tobytes() == hashlib.md5(pre[i].tobytes() + bufs[i].tobytes()).digest()


def test_packed_file_md5_matches_unpacked():
    """par2cuda_file_md5_packed (32 chains per warp) gives the same digests as
    the one-chain-per-block launch, for 40 uneven files including a 1-byte one."""
    torch = pytest.importorskip("torch")
    from parpar_gb300 import _lib
    from parpar_gb300.job import ResidentJob
    S = 4096
    rng = np.random.default_rng(40)
    lens = [int(x) for x in rng.integers(1, 40 * S, size=39)] + [1]
    job = ResidentJob(S, lens, [0])
    job.fill_synthetic(5)
    L = _lib.load()
    outs = []
    for fn in (L.par2cuda_file_md5, L.par2cuda_file_md5_packed):
        d = torch.zeros(16 * len(lens), dtype=torch.uint8, device="cuda")
        _lib.check(fn(job.d_in.data_ptr(), job.pitch, len(lens), job.d_flen.data_ptr(), job.d_first.data_ptr(), S,
                      d.data_ptr(), None), "md5")
        outs.append(d.cpu().numpy())
    assert np.array_equal(outs[0], outs[1])
    rows = job.d_in.view(torch.uint8).cpu().numpy()
    f = 7
    a = int(job.first_row[f])
    data = rows[a:a + (lens[f] + S - 1) // S, :S].reshape(-1)[:lens[f]]
    assert outs[0][16 * f:16 * f + 16].tobytes() == O.md5(data)


@pytest.mark.parametrize("S", [4, 60, 68, 72, 76, 1020, 4100, 8200, 12300, 20484])
def test_file_md5_of_rows_that_split_blocks(S):
    """Slice sizes of whole words that are no multiple of a 64-byte block: rows
    begin inside a block, at every 16-byte phase, with whole and partial last
    rows; one file per block, packed and pooled."""
    torch = pytest.importorskip("torch")
    L = _lib.load()
    lengths = [1, 63, 64, S - 1, S, S + 1, 2 * S + 3, 3 * S, 5 * S + S // 2, 9 * S - 2]
    files = [synth.slice_bytes(900 + S, k, n) for k, n in enumerate(lengths)]
    d, pitch, lens, first, nrows = _rows_from_files(torch, files, S)
    want = b"".join(hashlib.md5(f.tobytes()).digest() for f in files)
    flen = torch.tensor(lengths, dtype=torch.int64, device="cuda")
    d_first = torch.from_numpy(first.view(np.int32)).cuda()
    for call in (L.par2cuda_file_md5, L.par2cuda_file_md5_packed,
                 lambda *a: L.par2cuda_file_md5_pooled(*a[:7], 64, a[7])):
        md5 = torch.zeros(16 * len(files), dtype=torch.uint8, device="cuda")
        _lib.check(call(d.data_ptr(), pitch, len(files), flen.data_ptr(), d_first.data_ptr(), S, md5.data_ptr(), None), "file_md5")
        torch.cuda.synchronize()
        assert md5.cpu().numpy().tobytes() == want


@pytest.mark.parametrize("prefix", [0, 4, 8, 12, 16, 36, 60, 64, 100])
@pytest.mark.parametrize("data", [0, 27, 28, 60, 92, 128, 1000, 4097])
def test_rows_md5_prefixes(prefix, data):
    torch = pytest.importorskip("torch")
    L = _lib.load()
    n = 35
    pitch = L.par2cuda_row_pitch_bytes(max(data, 2))
    rows = synth.slices(77, 0, n, pitch)
    pre = synth.slices(78, 0, n, max(prefix, 1))[:, :prefix]
    d = torch.from_numpy(rows.copy()).cuda()
    d_pre = torch.from_numpy(np.ascontiguousarray(pre)).cuda() if prefix else None
    out = torch.zeros(16 * n, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_rows_md5(d.data_ptr(), pitch, n, data, d_pre.data_ptr() if prefix else None, prefix, out.data_ptr(),
                                   None), "rows_md5")
    torch.cuda.synchronize()
    want = b"".join(hashlib.md5(pre[i].tobytes() + rows[i, :data].tobytes()).digest() for i in range(n))
    assert out.cpu().numpy().tobytes() == want


@pytest.mark.parametrize("n", [1, 64, 65, 150])
def test_ifsc_lengths_around_the_crc_step(n):
    """Row lengths around the 512-byte step of the CRC and its four-step loop."""
    torch = pytest.importorskip("torch")
    L = _lib.load()
    S = 5000
    pitch = L.par2cuda_row_pitch_bytes(S)
    edges = [0, 1, 511, 512, 513, 1535, 2047, 2048, 2049, 2560, 4095, 4096, 4608, 4999, 5000]
    lens = np.array([edges[k % len(edges)] for k in range(n)], dtype=np.uint32)
    rows = synth.slices(79, 0, n, pitch)
    d = torch.from_numpy(rows.copy()).cuda()
    d_lens = torch.from_numpy(lens.view(np.int32)).cuda()
    out = torch.zeros(n * 20, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_slice_hash(d.data_ptr(), pitch, n, d_lens.data_ptr(), S, out.data_ptr(), None), "slice_hash")
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(n, 20)
    for i in range(n):
        padded = rows[i, :lens[i]].tobytes() + bytes(S - int(lens[i]))
        assert got[i].tobytes() == hashlib.md5(padded).digest() + zlib.crc32(padded).to_bytes(4, "little"), (i, lens[i])


@pytest.mark.parametrize("S", [4, 60, 64, 68, 128, 192, 196, 256, 1020, 1088])
def test_ifsc_partial_blocks_of_neighbouring_rows(S):
    """Rows of one warp that end in different blocks: an even and an odd number of blocks, with and without a remainder,
    each row's last block empty, begun, whole, or shared by a pair."""
    torch = pytest.importorskip("torch")
    L = _lib.load()
    n = 35                            # two blocks of 16 rows and a part of one
    pitch = L.par2cuda_row_pitch_bytes(S)
    lens = np.array([(S, 0, S - 1, 64 * (i % 5), 64 * (i % 7) + i, S // 2, 3 * i)[i % 7] for i in range(n)])
    lens = np.minimum(lens, S).astype(np.uint32)
    rows = synth.slices(80, 0, n, pitch)
    d = torch.from_numpy(rows.copy()).cuda()
    d_lens = torch.from_numpy(lens.view(np.int32)).cuda()
    out = torch.zeros(n * 20, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_slice_hash(d.data_ptr(), pitch, n, d_lens.data_ptr(), S, out.data_ptr(), None), "slice_hash")
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(n, 20)
    for i in range(n):
        padded = rows[i, :lens[i]].tobytes() + bytes(S - int(lens[i]))
        assert got[i].tobytes() == hashlib.md5(padded).digest() + zlib.crc32(padded).to_bytes(4, "little"), (i, lens[i])


@pytest.mark.parametrize("offset", [1, 2, 3, 4, 13])
@pytest.mark.parametrize("S", [100, 4100, 72, 33])
def test_file_md5_of_rows_at_any_address(S, offset):
    """Slice sizes that are no multiple of a 64-byte block: the rows may begin at any byte."""
    torch = pytest.importorskip("torch")
    L = _lib.load()
    lengths = [1, 63, 64, S - 1, S, S + 1, 2 * S + 3, 5 * S + S // 2]
    files = [synth.slice_bytes(700 + S, k, n) for k, n in enumerate(lengths)]
    d, pitch, lens, first, nrows = _rows_from_files(torch, files, S)
    moved = torch.zeros(d.numel() * d.element_size() + 16, dtype=torch.uint8, device="cuda")
    moved[offset:offset + moved.numel() - 16] = d.view(torch.uint8).reshape(-1)
    want = b"".join(hashlib.md5(f.tobytes()).digest() for f in files)
    flen = torch.tensor(lengths, dtype=torch.int64, device="cuda")
    d_first = torch.from_numpy(first.view(np.int32)).cuda()
    for call in (L.par2cuda_file_md5, L.par2cuda_file_md5_packed,
                 lambda *a: L.par2cuda_file_md5_pooled(*a[:7], 64, a[7])):
        md5 = torch.zeros(16 * len(files), dtype=torch.uint8, device="cuda")
        _lib.check(call(moved.data_ptr() + offset, pitch, len(files), flen.data_ptr(), d_first.data_ptr(), S, md5.data_ptr(),
                        None), "file_md5")
        torch.cuda.synchronize()
        assert md5.cpu().numpy().tobytes() == want


@pytest.mark.parametrize("n,S", [(10, 1020), (1340, 1024), (1341, 1024), (1085, 1500), (1086, 1500), (4031, 4096), (4032, 4096),
                                 (8192, 24576), (8193, 24576), (32768, 68)])
def test_ifsc_of_short_and_many_rows(n, S):
    """Both sides of the row counts at which one thread per row takes over, with full, short, empty and odd rows."""
    torch = pytest.importorskip("torch")
    L = _lib.load()
    pitch = L.par2cuda_row_pitch_bytes(S)
    lens = np.array([(S, S - 1, 0, 64 * (i % (S // 64 + 1)), i % (S + 1))[i % 5] for i in range(n)], dtype=np.uint32)
    rows = synth.slices(82, 0, n, pitch)
    d = torch.from_numpy(rows.copy()).cuda()
    d_lens = torch.from_numpy(lens.view(np.int32)).cuda()
    out = torch.zeros(n * 20, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_slice_hash(d.data_ptr(), pitch, n, d_lens.data_ptr(), S, out.data_ptr(), None), "slice_hash")
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(n, 20)
    for i in range(n):
        padded = rows[i, :lens[i]].tobytes() + bytes(S - int(lens[i]))
        assert got[i].tobytes() == hashlib.md5(padded).digest() + zlib.crc32(padded).to_bytes(4, "little"), (i, lens[i])


@pytest.mark.parametrize("offset", [1, 2, 3, 4, 13])
@pytest.mark.parametrize("S", [4, 33, 63, 2000])
def test_ifsc_of_short_rows_at_any_address(S, offset):
    """Rows of less than a block may begin at any byte."""
    torch = pytest.importorskip("torch")
    L = _lib.load()
    n, pitch = 35, 64
    lens = np.array([(S, 0, S - 1, S // 2, i % S)[i % 5] for i in range(n)], dtype=np.uint32) % 64
    rows = synth.slices(81, 0, n, pitch)
    d = torch.zeros(n * pitch + 16, dtype=torch.uint8, device="cuda")
    d[offset:offset + n * pitch] = torch.from_numpy(rows.reshape(-1).copy()).cuda()
    d_lens = torch.from_numpy(lens.view(np.int32)).cuda()
    out = torch.zeros(n * 20, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_slice_hash(d.data_ptr() + offset, pitch, n, d_lens.data_ptr(), S, out.data_ptr(), None), "slice_hash")
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(n, 20)
    for i in range(n):
        padded = rows[i, :lens[i]].tobytes() + bytes(S - int(lens[i]))
        assert got[i].tobytes() == hashlib.md5(padded).digest() + zlib.crc32(padded).to_bytes(4, "little"), (i, lens[i])


@pytest.mark.parametrize("n", [4864, 4865, 9728, 9729, 9800])
@pytest.mark.parametrize("prefix", [0, 36, 64])
def test_rows_md5_of_many_rows(n, prefix):
    """Both sides of the row counts at which a warp takes more rows."""
    torch = pytest.importorskip("torch")
    L = _lib.load()
    data, pitch = 200, 256
    rows = synth.slices(83, 0, n, pitch)
    pre = synth.slices(84, 0, n, max(prefix, 2))[:, :prefix]
    d = torch.from_numpy(rows.copy()).cuda()
    d_pre = torch.from_numpy(np.ascontiguousarray(pre)).cuda() if prefix else None
    out = torch.zeros(16 * n, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_rows_md5(d.data_ptr(), pitch, n, data, d_pre.data_ptr() if prefix else None, prefix, out.data_ptr(),
                                   None), "rows_md5")
    torch.cuda.synchronize()
    want = b"".join(hashlib.md5(pre[i].tobytes() + rows[i, :data].tobytes()).digest() for i in range(n))
    assert out.cpu().numpy().tobytes() == want


@pytest.mark.parametrize("per", [32, 64])
@pytest.mark.parametrize("n", [31, 65, 4864, 4865])
def test_staged_file_md5_of_many_files(n, per):
    """Both sides of the file count at which a warp takes more files, and part-filled blocks."""
    torch = pytest.importorskip("torch")
    L = _lib.load()
    S, pitch = 64, 128
    lens = np.array([(1, 63, 64, 65, 128, 150)[i % 6] for i in range(n)], dtype=np.int64)
    first = np.concatenate(([0], np.cumsum((lens + S - 1) // S)[:-1])).astype(np.int32)
    rows = synth.slices(85, 0, int(first[-1]) + 3, pitch)
    d = torch.from_numpy(rows.copy()).cuda()
    d_len, d_first = torch.from_numpy(lens).cuda(), torch.from_numpy(first).cuda()
    out = torch.zeros(16 * n, dtype=torch.uint8, device="cuda")
    _lib.check(L.par2cuda_file_md5_staged(d.data_ptr(), pitch, n, d_len.data_ptr(), d_first.data_ptr(), S, out.data_ptr(), per,
                                          None), "staged")
    torch.cuda.synchronize()
    assert L.par2cuda_device_error() == 0
    want = b"".join(hashlib.md5(rows[first[i]:first[i] + 3, :S].tobytes()[:lens[i]]).digest() for i in range(n))
    assert out.cpu().numpy().tobytes() == want
