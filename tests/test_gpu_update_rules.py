"""The update rules and constraints that take a path of their own in the row
passes (flipping positivity, ER), in every family of passes, against the oracle,
bit for bit: the operations are the oracle's in its order, so no tolerance
applies."""
import numpy as np
import pytest

from tests._engines import AREA, ER, HIO, RAAR, same_bits, setup

pytestmark = pytest.mark.gpu

PERSIST = 4  # SPB_TUNE_PERSIST
# 8 points a thread, 16 points a thread, a persistent block a start, mixed-radix
# with and without a prime step
SHAPES = [((256, 256), 0), ((128, 64), 0), ((64, 64), 2), ((45, 50), 0), ((30, 28), 0)]


@pytest.mark.parametrize("shape,persist", SHAPES)
@pytest.mark.parametrize("alg,cons", [(HIO, 2 | 8), (RAAR, 4 | 8), (ER, 4 | 8), (RAAR, 1 | 8), (HIO, 8), (ER, 0)])
def test_flipping_positivity_and_er(lib, oracle_mod, shape, persist, alg, cons):
    sup = [(AREA, 5, 2.0, 0.1)]
    ref = setup(oracle_mod.Restatement(shape), shape, alg, sup, constraints=cons)
    gpu = setup(lib.Phaser(shape), shape, alg, sup, constraints=cons)
    gpu.set_tuning(PERSIST, persist)
    for n in (1, 11):
        assert ref.iterate(n) == 0 and gpu.iterate(n) == 0
        for which in (0, 1, 2):
            assert same_bits(gpu.get(which), ref.get(which)), (n, which)
        assert np.array_equal(gpu.flags(), ref.flags())
    gpu.close()


@pytest.mark.parametrize("mode", ["margins", "phased"])
@pytest.mark.parametrize("shape", [(45, 66), (37, 192), (14, 20, 9)])
def test_projections_pixel_by_pixel(lib, oracle_mod, mode, shape):
    """Amplitude margins and phased amplitudes, in columns that end mid-group."""
    rng = np.random.default_rng(4)
    amp = np.abs(rng.standard_normal(shape)).astype(np.float32) * 20
    ref, gpu = (setup(e, shape, HIO, None, constraints=2 | (32 if mode == "margins" else 0))
                for e in (oracle_mod.Restatement(shape), lib.Phaser(shape)))
    lo, hi = (amp * 0.8).astype(np.float32), (amp * 1.1).astype(np.float32)
    phased = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    mask = (rng.random(shape) < 0.7).astype(np.int32)
    for e in (ref, gpu):
        if mode == "margins":
            e.set_amplitudes(amp, mask)
            e.set_amplitudes_margins(lo, hi)
        else:
            e.set_phased_amplitudes(phased, mask)
            e.set_objective(1)
        assert e.iterate(5) == 0
    assert same_bits(gpu.model(), ref.model())
    gpu.close()


@pytest.mark.parametrize("shape", [(9, 14, 22), (5, 13, 67), (3, 1, 30), (8, 35, 16)])
def test_blur_of_ragged_volumes(lib, oracle_mod, shape):
    rng = np.random.default_rng(2)
    x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    assert same_bits(lib.gaussian_blur(x, 1.7), oracle_mod.gaussian_blur(x, 1.7))
