"""The persistent form of the split-BF16 SGEMM (one CTA per SM walking several
tiles), which hml_sgemm_ex runs whole-K configurations of several waves of row
tiles with (GPU).

Every result must equal, bit for bit, what the configuration itself gives
(hml_sgemm_ex_config), except the rows of a last wave that is split in K, which
must equal the same tile split that many ways; repeated calls give the same
bits.  Shapes: every tile width, both orders of A, whole waves only, a last wave
too full to split, split tails down to one tile, K shorter than a chunk and not
a multiple of one, several column tiles, a ragged last row tile.
"""
import os

import pytest

import hiperml_b200 as hml

pytestmark = pytest.mark.gpu
VAR = {16: 0, 32: 1, 64: 2, 128: 3}


def select(tmp_path, akc, bkc, M, N, K, cfg):
    f = tmp_path / "tuned.txt"
    f.write_text("#HML-B200 tuning v2\n# device test sms 148\n"
                 "# akc bkc M N K : algo tile_m tile_n split_k stages variant time_us\n"
                 "%d %d %d %d %d : %s 1.0\n" % (akc, bkc, M, N, K,
                                              " ".join(str(v) for v in cfg.as_tuple())))
    hml.tune_clear()
    assert hml.tune_load(str(f)) == 1


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("bn,waves,rest,N,K", [
    (32, 2, 0, 32, 256), (32, 2, 100, 27, 320), (32, 2, 1, 32, 1024), (16, 2, 30, 16, 4096),
    (64, 3, 70, 64, 2048), (128, 2, 74, 128, 1088), (32, 5, 20, 20, 32), (32, 2, 7, 32, 36),
    (64, 1, 74, 50, 1000), (128, 2, 11, 300, 200), (16, 3, 148, 16, 68)])
def test_persistent_bits(cuda, tmp_path, ta, bn, waves, rest, N, K):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = waves * sms + rest
    cols = -(-N // bn)
    M = (tiles // cols) * 128 - 37  # a ragged last row tile
    M -= M % 4                      # addressable either way
    cfg = hml.SgemmConfig(hml.ALGO_BF16X6, 128, bn, 1, 6, VAR[bn])
    A = torch.empty(M * K, device="cuda")
    B = torch.empty(K * N, device="cuda")
    hml.fill_random(A, 5, 0, 1)
    hml.fill_random(B, 5, 1, 1)
    lda = K if ta else M

    def run(config=None):
        C = torch.full((M * N,), 0.5, device="cuda")
        hml.sgemm_ex(0, ta, 0, M, N, K, 1.5, A, lda, B, K, -2.0, C, M, config=config)
        return C.view(N, M)

    try:
        select(tmp_path, ta, 1, M, N, K, cfg)
        assert hml.select(0, ta, 0, M, N, K).as_tuple() == cfg.as_tuple()
        got = run()
        for _ in range(3):
            assert torch.equal(got, run())
        whole = run(cfg)
        row_tiles = -(-M // 128)
        tail = row_tiles % sms if cols == 1 else 0
        split = 1
        if tail and 2 * tail <= sms:
            while split < 8 and 2 * split * tail <= sms and -(-K // 64) * 64 // (2 * split) >= 256:
                split *= 2
        m1 = (row_tiles - tail) * 128 if split > 1 else M
        assert torch.equal(got[:, :m1], whole[:, :m1])
        if split > 1:
            sk = run(hml.SgemmConfig(hml.ALGO_BF16X6, 128, bn, split, 6, VAR[bn]))
            assert torch.equal(got[:, m1:], sk[:, m1:])
        assert hml.device_error() == 0
    finally:
        hml.tune_clear()
        hml.tune_load(os.path.join(os.path.dirname(hml.__file__), "data", "tuned_b200.txt"))


def test_persistent_graph(cuda):
    """Captured and replayed, the tail's counters are ready for every replay."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    M, N, K = (2 * sms + 20) * 128, 32, 1024
    A = torch.empty(K, M, device="cuda").uniform_(-1, 1)
    B = torch.empty(N, K, device="cuda").uniform_(-1, 1)
    C = torch.zeros(N, M, device="cuda")
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        hml.sgemm_ex(0, 0, 0, M, N, K, 1.0, A, M, B, K, 0.0, C, M)
        want = C.clone()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for _ in range(2):
                hml.sgemm_ex(0, 0, 0, M, N, K, 1.0, A, M, B, K, 0.0, C, M)
        for _ in range(5):
            C.zero_()
            g.replay()
            assert torch.equal(C, want)
