"""Packing at the edges of its tiles: read lengths around whole words and
16-byte groups, counts around a tile's reads, buffers that start at any byte,
N, lower case and other letters, against a numpy restatement (whole words)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 2, 16, 17, 31, 32, 33, 37, 75, 101, 150, 151, 251, 300, 512])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 127, 128, 129, 3000])
def test_pack(L, n):
    import torch
    from curc_b200 import Context
    rng = np.random.default_rng([L, n])
    reads = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, size=(n, L))].copy()
    m = rng.random((n, L))
    reads[m < 0.003] = ord("N")
    reads[(m > 0.003) & (m < 0.005)] = ord("R")
    reads[(m > 0.005) & (m < 0.010)] |= 0x20
    code = np.zeros(256, np.uint64)
    for c, v in zip(b"ACGTacgt", [0, 1, 2, 3, 0, 1, 2, 3]):
        code[c] = v
    W = (L + 31) // 32
    codes = np.zeros((n, W * 32), np.uint64)
    codes[:, :L] = code[reads]
    want = (codes.reshape(n, W, 32) << (62 - 2 * np.arange(32)).astype(np.uint64)).sum(axis=2, dtype=np.uint64)
    want_n = (reads == ord("N")).any(axis=1).astype(np.uint8)
    flat = torch.from_numpy(reads.reshape(-1)).cuda()
    with Context(0) as ctx:
        for skew in (0, 1, 2, 3, 8):  # bytes before the first read
            buf = torch.zeros(n * L + 16, dtype=torch.uint8, device="cuda")
            buf[skew:skew + n * L] = flat
            packed = torch.full((n, W), -1, dtype=torch.int64, device="cuda")
            has_n = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            ctx.pack_device(buf.data_ptr() + skew, n, L, packed.data_ptr(), has_n.data_ptr())
            assert np.array_equal(packed.cpu().numpy().view(np.uint64), want), skew
            assert np.array_equal(has_n.cpu().numpy(), want_n), skew
