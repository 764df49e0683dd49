"""Two runs per warp (dims 1 to 4) in requests that fill the GPU, where the default packs too: both register budgets of
the mixed kernel, all models, odd run counts, either run of a pair, and FP64 digits at every chunk length and digit
scale.  Below that size a request runs packed only if its caller says so."""
import numpy as np
import pytest

from conftest import normwise_err

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
def test_mixed_shapes_give_the_same_bits(jne, dim):
    n = 16 * _sms() + 35
    with jne.Engine(0) as eng:
        for model in range(5):
            few = np.concatenate([eng.eigs_seeded(model, dim, 1000, 7 + a, min(900, n - a), precision=jne.PREC_MIXED)
                                  for a in range(0, n, 900)])  # unpacked by default
            by_default = eng.eigs_seeded(model, dim, 1000, 7, n, precision=jne.PREC_MIXED)
            assert np.array_equal(by_default, few), model
            with jne.Engine(0) as shaped:
                for bps in (4, 6):
                    for pack in (1, 0):
                        shaped.set_launch_shape(bps, pack)
                        for count in (1, 2, 333, n):
                            got = shaped.eigs_seeded(model, dim, 1000, 7, count, precision=jne.PREC_MIXED)
                            assert np.array_equal(got, few[:count]), (model, bps, pack, count)


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("bps", [4, 6])
def test_mixed_packed_against_fp64_and_the_partner(jne, dim, bps):
    with jne.Engine(0) as eng:
        eng.set_launch_shape(bps, 1)
        for model in (0, 3, 4):
            full = eng.eigs_seeded(model, dim, 1500, 11, 333, precision=jne.PREC_MIXED)
            shifted = eng.eigs_seeded(model, dim, 1500, 12, 332, precision=jne.PREC_MIXED)  # the other pairs
            assert np.array_equal(full[1:], shifted), model
            fp64 = eng.eigs_seeded(model, dim, 1500, 11, 333, precision=jne.PREC_FP64)
            assert normwise_err(full, fp64, 1.0) < 2e-6, model  # the mixed bound of test_packing_gpu.py


@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("steps", [33, 300, 512, 513, 1100, 2048, 2049, 2500])
def test_digits_packed(engine, jne, dim, steps):
    n = 80 * _sms() + 35  # above the line at every length
    for model in range(5):
        few = np.concatenate([engine.eigs_seeded(model, dim, steps, 5 + a, min(1800, n - a), precision=jne.PREC_FP64)
                              for a in range(0, n, 1800)])
        packed = engine.eigs_seeded(model, dim, steps, 5, n, precision=jne.PREC_FP64)
        assert np.array_equal(packed, few), model
        other = engine.eigs_seeded(model, dim, steps, 6, n - 1, precision=jne.PREC_FP64)  # the other pairs
        assert np.array_equal(other, packed[1:]), model
    dB, _ = engine.export_increments(dim, steps, 5, 64)
    ref = engine.eigs_from_increments(4, dB, precision=jne.PREC_FP64)
    assert normwise_err(packed[:64], ref) < 1e-10  # as in test_digits_gpu.py
