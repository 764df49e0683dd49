"""FP64 runs whose walk passes the digit limit (6.8 standard deviations of a full chunk) inside a chunk, which then ends
early: seeds found by searching the streams (a few in 10^11 first chunks; dim 12: features 8 to 11, block 1's columns).
Their eigenvalues against the general path, and their bits and their pair's alone, packed as either run of a pair,
and just past the end of an odd request.

Tolerance against the general path: T 2^-53 relative to a moment, amplified by the pencil's condition, as in
test_digits_gpu.py."""
import numpy as np
import pytest

from conftest import normwise_err

pytestmark = pytest.mark.gpu

# (dim, base seed, run seed): |W| 169 at step 480; 160 at 448; 161; 156; -155 at 480 after 161 at 448; 156
HITS = [(4, 1033, 839867243), (4, 1037, 3131208496), (4, 1063, 1216090068), (4, 1084, 961007897),
        (12, 1043, 3370578285), (12, 1051, 2792512970)]


@pytest.mark.parametrize("dim,base,seed", HITS)
def test_the_walk_passes_the_limit(engine, dim, base, seed):
    dB, _ = engine.export_increments(dim, 2100, seed, 1, base_seed=base)
    z = (dB[0, :480] * np.sqrt(2100)).astype(np.float32).astype(float)
    assert (np.abs(np.cumsum(z, axis=0)[31:480:32]) > 155).any()  # at a tile's end: steps 32 .. 480


@pytest.mark.parametrize("dim,base,seed", HITS)
@pytest.mark.parametrize("steps", [2049, 2100, 4500])
def test_early_chunk_ends_against_the_general_path(engine, jne, dim, base, seed, steps):
    dB, _ = engine.export_increments(dim, steps, seed - 1, 3, base_seed=base)
    for model in range(5):
        ref = engine.eigs_from_increments(model, dB, precision=jne.PREC_FP64)
        got = engine.eigs_seeded(model, dim, steps, seed - 1, 3, precision=jne.PREC_FP64, base_seed=base)
        assert normwise_err(got, ref) < 1e-10, model


@pytest.mark.parametrize("dim,base,seed", [h for h in HITS if h[0] <= 4])
def test_a_pair_with_an_early_end_keeps_each_runs_bits(engine, jne, dim, base, seed):
    import torch

    line = 80 * torch.cuda.get_device_properties(0).multi_processor_count  # packed above
    for model in (0, 3, 4):
        alone = {s: engine.eigs_seeded(model, dim, 2100, s, 1, precision=jne.PREC_FP64, base_seed=base)[0]
                 for s in range(seed - 2, seed + 3)}
        for before in (100, 101):  # the run as first and as second of its pair
            n = line + 35
            got = engine.eigs_seeded(model, dim, 2100, seed - before, n, precision=jne.PREC_FP64, base_seed=base)
            for s, want in alone.items():
                assert np.array_equal(got[before + s - seed], want), (model, before, s - seed)
        n = line + 1 + line % 2  # odd: the last unit's second run is past the request
        for past in (0, 1):
            got = engine.eigs_seeded(model, dim, 2100, seed - n + 1 - past, n, precision=jne.PREC_FP64, base_seed=base)
            assert np.array_equal(got[-1], alone[seed - past]), (model, past)
