"""Passes with compile-time plans (192, 384 and 1000-point lines, on the grids
that they are chosen for) against the oracle, bit for bit: the operations are
the oracle's in its order, so no tolerance applies."""
import numpy as np
import pytest

from tests._engines import AREA, DIFFMAP, ER, HIO, RAAR, THRESHOLD, same_bits, setup

pytestmark = pytest.mark.gpu

# rows and columns of each length alone and together, one to three rows a block
# and a part of one, columns that do not fill a block, every update rule and
# constraint (1 real, 2 positive, 4 positive complex, 8 flipping, 16
# centrosymmetric), and grids on the other side of the choice
RUNS = [
    ((192, 37), HIO, 2), ((37, 192), RAAR, 4), ((598, 192), ER, 2 | 8), ((890, 192), HIO, 1), ((1190, 192), RAAR, 0),
    ((384, 30), HIO, 2 | 16), ((30, 384), ER, 1), ((384, 192), RAAR, 2), ((192, 384), HIO, 4 | 8), ((600, 384), HIO, 2),
    ((1000, 22), RAAR, 2), ((1000, 600), HIO, 0), ((1000, 1190), HIO, 2), ((5, 192, 6), HIO, 2), ((192, 5, 7), RAAR, 1),
    ((384, 3, 4), ER, 2), ((192, 6, 5), DIFFMAP, 16), ((1000, 3, 2), DIFFMAP, 2), ((1190, 1000), DIFFMAP, 2),
    ((1000, 1190), DIFFMAP, 16),
]


@pytest.mark.parametrize("shape,alg,cons", RUNS)
def test_iterations(lib, oracle_mod, shape, alg, cons):
    sup = [(AREA, 4, 2.0, 0.1)] if alg != RAAR else [(THRESHOLD, 4, 2.0, 0.2)]
    ref = setup(oracle_mod.Restatement(shape, threads=8), shape, alg, sup, constraints=cons)
    gpu = setup(lib.Phaser(shape), shape, alg, sup, constraints=cons)
    for n in (1, 6):
        assert ref.iterate(n) == 0 and gpu.iterate(n) == 0
        for which in (0, 1, 2):
            assert same_bits(gpu.get(which), ref.get(which)), (n, which)
        assert np.array_equal(gpu.flags(), ref.flags())
    gpu.close()


@pytest.mark.parametrize("shape,starts", [((192, 192), 7), ((384, 384), 3), ((192, 384), 4)])
def test_starts_follow_one_another(lib, oracle_mod, shape, starts):
    from libspimage_b200 import synth

    amp, mask, support, _ = synth.small_pattern(shape, seed=1)
    seeds = list(range(3, 3 + starts))
    gpu = lib.Phaser(shape)
    gpu.set_algorithm(HIO, beta=0.9, constraints=2)
    gpu.add_support_update(AREA, 4, 2.0, 0.1)
    gpu.start()
    gpu.set_starts(starts)
    gpu.set_amplitudes(amp, mask)
    assert gpu.init_models(1, seeds) == 0
    gpu.set_support(support)
    assert gpu.iterate(7) == 0
    for b in (0, starts - 1):
        ref = setup(oracle_mod.Restatement(shape, threads=8), shape, HIO, [(AREA, 4, 2.0, 0.1)], seed=seeds[b])
        assert ref.iterate(7) == 0
        assert same_bits(gpu.start_model(b), ref.model()), b
    gpu.close()
