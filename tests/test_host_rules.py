"""Rules that the host decides by (which launches a step is cut into, which kernel takes it), without a GPU."""


def test_runs_of_chunks():
    """Launches of at most so many chunks hold every chunk of every sequence once and in order, and leave whole what fits."""
    from airframe_b200.kernels import _chunk_runs
    for lens in ([1], [32], [33], [500], [40, 300, 1, 224, 64], [32] * 7, [1, 1, 1], [96, 97, 95]):
        chunks = [-(-n // 32) for n in lens]
        owner = [s for s, c in enumerate(chunks) for _ in range(c)]
        for most in (1, 2, 3, 5, 512):
            runs = _chunk_runs(lens, 32, most)
            at = 0
            for s0, seqs, c0, count in runs:
                assert c0 == at and 0 < count <= most and owner[c0:c0 + count] == sorted(owner[c0:c0 + count])
                assert sorted(set(owner[c0:c0 + count])) == list(range(s0, s0 + seqs))
                at += count
            assert at == len(owner)
            for s, c in enumerate(chunks):
                met = sum(s0 <= s < s0 + seqs for s0, seqs, _, _ in runs)
                assert met == -(-c // most)


def test_which_steps_go_in_chunks():
    """Steps whose recurrence is faster in chunks, and steps whose chunks would be mostly empty (measured: see the rule)."""
    from airframe_b200.parts.recurrent import chunks_pay
    for lens in ([128], [129], [2048], [128] * 16, [160] * 64, [129] * 8, [128, 40] * 8, [512] + [8] * 15, [2048] + [1] * 16, [2048] + [1] * 64,
                 [130] + [40] * 63, [513] * 4):
        assert chunks_pay(lens), lens
    for lens in ([1], [127], [64] * 16, [33] * 16, [128] + [1] * 63, [128] + [1] * 255, [128] + [8] * 60, [130] + [17] * 63, [2048] + [1] * 400):
        assert not chunks_pay(lens), lens


def test_attention_of_prompts_in_32_bits_takes_rows_of_one_number():
    """Keys or values of fewer rows than the queries are refused before anything is launched: the kernel would read behind them."""
    import pytest
    import torch
    from airframe_b200 import kernels
    q, short, starts = torch.zeros(80, 64), torch.zeros(79, 64), torch.tensor([0, 80], dtype=torch.int32)
    for k, v in ((short, q), (q, short)):
        with pytest.raises(kernels.KernelError, match="the same rows"):
            kernels.attn_prefill_f32(torch.zeros(80, 64), q, k, v, starts, 1, 80, 1, 1, 64, 1.0, 0.0, 0)
