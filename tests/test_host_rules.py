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
