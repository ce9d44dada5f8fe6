"""A warp that has seen the failure limit takes no new realisation, also for the
lanes whose paths were still under way when it saw it. One warp: it looks at
every 4th fetch, its first failure comes with the first fetch, and a fetch takes
at most 32 realisations, so it runs at most 4 x 32. Paths fail at once over one
plate and bounce 65 times and more between two facing mirrors beside it, so that
lanes are under way at every fetch."""
import pytest

import pyssol as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trap", [3.0, 5.0, 8.0])
def test_no_realisation_after_the_limit(product, trap):
    s = P.Scene(product)
    air, glass = s.medium(0.0, 1.0), s.medium(0.0, 1.5)
    wrong, v, m = s.dielectric(glass, air), s.virtual(), s.mirror(1.0, 0.0)
    # rays from the air meet a plate whose outside is glass: a failure
    s.instance(s.object([(s.rectangle(5, 5), v, v)]), P.transform_from(None, (0, 0, 2.0)))
    s.instance(s.object([(s.rectangle(5, 5), wrong, wrong)]),
               P.transform_from(None, (0, 0, 1.0)), sample=0)
    # mirrors face to face, the upper one open to the sun on its back
    half = trap / 2
    s.instance(s.object([(s.rectangle(half, half), m, m)]), P.transform_from(None, (30, 0, 0)))
    s.instance(s.object([(s.rectangle(half, half), m, v)]),
               P.transform_from(P.rotation_pitch_pi(), (30, 0, 1.0)), sample=0)
    s.set_sun("directional", (0, 0, -1), 1000.0)
    opt = P.options()
    opt.block_size, opt.grid_blocks = 32, 1
    ran = []
    for seed in range(6):
        e = s.solve(100000, seed=seed, max_failed=1, options=opt, check=False)
        assert e.res == P.RES_BAD_OP
        ran.append(e.count("failed_count") + e.count("realisation_count"))
    assert max(ran) <= 128, ran
