"""How the 32-bit product is cut into runs, tiles and clusters: the rule alone, on the CPU."""
import ctypes

import pytest

GROUPS, SHORTEST, STAGE = 8, 128, 32


@pytest.fixture(scope="module")
def plan():
    from alpacca_b200.ops import build
    lib = build.load("gemm_f32")

    def call(M, N, K):
        out = (ctypes.c_int * 4)()
        lib.ab_gemm_f32_plan(M, N, K, out)
        return tuple(out)
    return call


KS = [1, 32, 96, 128, 129, 200, 224, 256, 384, 385, 512, 513, 704, 768, 896, 1024, 1100, 1120, 1600, 2048, 3000, 8192, 14336]


@pytest.mark.parametrize("K", KS)
def test_every_processor_of_a_tile_has_a_run(plan, K):
    """No cluster has a member without k, members cover all runs, and the sums have room in tensor memory."""
    for N in (1, 64, 130, 2048, 3072, 16384, 128256):
        for M in (1, 8, 16, 17, 32, 33, 48, 64, 65, 96, 100, 200, 333, 1000, 2048):
            run, n, per, cs = plan(M, N, K)
            runs = -(-K // run)
            assert run % STAGE == 0 and run >= SHORTEST and runs <= GROUPS, (M, N, K)
            assert n % 16 == 0 and 16 <= n <= 128 and per in (1, 4, 8) and 1 <= cs <= GROUPS, (M, N, K)
            assert cs * per * run >= K and (cs - 1) * per * run < K, (M, N, K, run, per, cs)
            assert (cs > 1) == (per < GROUPS), (M, N, K)
            assert n * (3 if runs == 1 else 4 if runs <= 4 or per < GROUPS else 5) <= 512, (M, N, K)


@pytest.mark.parametrize("M,N,K,longest", [(1, 2048, 256, 4), (1, 2048, 384, 4), (1, 2048, 768, 4), (1, 2048, 1100, 5), (8, 512, 896, 4),
                                           (200, 2048, 256, 4), (200, 2048, 768, 4), (1, 2048, 2048, 8)])
def test_few_tiles_share_their_runs(plan, M, N, K, longest):
    """Where tiles are few, no processor takes more than one run (in stages of k)."""
    run, _, per, cs = plan(M, N, K)
    assert min(K, run * per) <= longest * STAGE and cs == -(-K // run)
