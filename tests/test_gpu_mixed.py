"""Mixed-radix passes (lines without a register kernel of their own) against
the oracle, bit for bit: the device transform and pointwise steps are the
oracle's operations in the oracle's order, so no tolerance applies."""
import numpy as np
import pytest

from tests._engines import AREA, DIFFMAP, ER, HIO, RAAR, THRESHOLD, same_bits, setup

pytestmark = pytest.mark.gpu

# single steps, pairs of stages run as one, primes alone, repeated, first and
# last, the padded and unpadded first step, the longest lines
LENGTHS = [2, 3, 6, 7, 9, 10, 12, 14, 15, 22, 35, 45, 67, 75, 96, 121, 130, 225, 243, 257, 335, 600, 625, 768, 1021, 1331,
           2401, 3125, 7000, 7266, 8190, 8191]


@pytest.mark.parametrize("n", LENGTHS)
def test_transform_rows_and_columns(lib, oracle_mod, n):
    rng = np.random.default_rng(n)
    for shape in ((3, n), (n, 3)):
        x = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
        x.flat[:: max(2, n // 3)] = complex(-0.0, 0.0)  # signed zeros travel too
        for sign in (-1, 1):
            assert same_bits(lib.fft(x, sign), oracle_mod.fft(x, sign)), (shape, sign)


# grids of one wave and of many, columns that do not fill a block, odd rows,
# every update rule and constraint (1 real, 2 positive, 4 positive complex,
# 8 flipping, 16 centrosymmetric)
RUNS = [
    ((33, 35), HIO, 0), ((35, 33), RAAR, 1), ((130, 66), RAAR, 2), ((67, 75), HIO, 4), ((96, 90), ER, 2 | 8),
    ((45, 121), ER, 4 | 8), ((243, 100), HIO, 2 | 16), ((192, 330), RAAR, 2), ((35, 45), DIFFMAP, 2), ((64, 48), DIFFMAP, 1),
    ((7, 10, 15), HIO, 2), ((14, 9, 22), DIFFMAP, 0), ((60, 45, 48), RAAR, 2), ((16, 33, 12), ER, 1),
]


@pytest.mark.parametrize("shape,alg,cons", RUNS)
def test_iterations(lib, oracle_mod, shape, alg, cons):
    sup = [(AREA, 6, 2.0, 0.1)] if alg != RAAR else [(THRESHOLD, 6, 2.0, 0.2)]
    ref = setup(oracle_mod.Restatement(shape), shape, alg, sup, constraints=cons)
    gpu = setup(lib.Phaser(shape), shape, alg, sup, constraints=cons)
    for n in (1, 13):
        assert ref.iterate(n) == 0 and gpu.iterate(n) == 0
        for which in (0, 1, 2):
            assert same_bits(gpu.get(which), ref.get(which)), (n, which)
        assert np.array_equal(gpu.flags(), ref.flags())
    gpu.close()


@pytest.mark.parametrize("case", ["tiny", "zero model"])
def test_projection_outside_the_branch_free_domains(lib, oracle_mod, case):
    """Amplitudes below 2^-60, and a spectrum of zeros, take the IEEE forms."""
    shape = (45, 50)
    ref, gpu = (setup(e, shape, HIO, None) for e in (oracle_mod.Restatement(shape), lib.Phaser(shape)))
    amp = np.abs(np.random.default_rng(1).standard_normal(shape)).astype(np.float32)
    if case == "tiny":
        amp[3:9] *= np.float32(1e-25)
    for e in (ref, gpu):
        e.set_amplitudes(amp, np.ones(shape, np.int32))
        if case == "zero model":
            e.set_model(np.zeros(shape, np.complex64))
        assert e.iterate(5) == 0
    assert same_bits(gpu.model(), ref.model())
    gpu.close()


def test_batch_of_ragged_frames(lib, oracle_mod):
    """Starts follow one another in rows and columns without touching."""
    shape, seeds = (35, 66), [3, 9, 4, 7, 5]
    from libspimage_b200 import synth

    amp, mask, support, _ = synth.small_pattern(shape, seed=1)
    gpu = lib.Phaser(shape)
    gpu.set_algorithm(RAAR, beta=0.9, constraints=2)
    gpu.add_support_update(AREA, 6, 2.0, 0.1)
    gpu.start()
    gpu.set_starts(len(seeds))
    gpu.set_amplitudes(amp, mask)
    assert gpu.init_models(1, seeds) == 0
    gpu.set_support(support)
    assert gpu.iterate(14) == 0
    for b, s in enumerate(seeds):
        ref = setup(oracle_mod.Restatement(shape), shape, RAAR, [(AREA, 6, 2.0, 0.1)], seed=s)
        assert ref.iterate(14) == 0
        assert same_bits(gpu.start_model(b), ref.model()), b
    gpu.close()


# the difference map's two projections in one launch: 8-point lines (256, 512)
# and mixed-radix lines, with and without the Fourier constraint that only the
# first of the two takes; 1024-point lines keep two launches
@pytest.mark.parametrize("shape", [(256, 70), (512, 33), (45, 66), (1024, 24)])
@pytest.mark.parametrize("cons,starts", [(2, 1), (16, 1), (1, 3)])
def test_difference_map_projection_pair(lib, oracle_mod, shape, cons, starts):
    from libspimage_b200 import synth

    amp, mask, support, _ = synth.small_pattern(shape, seed=1)
    seeds = list(range(5, 5 + starts))
    gpu = lib.Phaser(shape)
    gpu.set_algorithm(DIFFMAP, beta=0.8, constraints=cons)
    gpu.start()
    gpu.set_starts(starts)
    gpu.set_amplitudes(amp, mask)
    assert gpu.init_models(1, seeds) == 0
    gpu.set_support(support)
    assert gpu.iterate(1) == 0 and gpu.iterate(5) == 0
    for b, seed in enumerate(seeds):
        ref = setup(oracle_mod.Restatement(shape), shape, DIFFMAP, None, constraints=cons, beta=0.8, seed=seed)
        assert ref.iterate(6) == 0
        assert same_bits(gpu.start_model(b), ref.model()), b
    gpu.close()


# several waves of the projection pass: the instance with fewer registers
@pytest.mark.parametrize("shape,alg", [((1024, 1536), RAAR), ((2048, 1024), HIO)])
def test_projection_pass_of_several_waves(lib, oracle_mod, shape, alg):
    ref, gpu = (setup(e, shape, alg, [(AREA, 4, 2.0, 0.1)]) for e in (oracle_mod.Restatement(shape, threads=8), lib.Phaser(shape)))
    assert ref.iterate(6) == 0 and gpu.iterate(6) == 0
    assert same_bits(gpu.model(), ref.model())
    assert np.array_equal(gpu.flags(), ref.flags())
    gpu.close()
