"""The host-side plans of the kernels (the matrix product: which side the tokens go on, the N
tile, the K split; the sampling kernel: CTAs per row): decisions only, no GPU.  The library is built by nvcc on first use."""
import ctypes
import shutil

import pytest


@pytest.fixture(scope="module")
def plan():
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc to build the kernel library with")
    from zinfer_b200 import ops

    lib = ops.lib()

    def f(M, N, K, sms=148):
        out = (ctypes.c_int * 3)()
        need = lib.zi_gemm_tcgen05_plan(M, N, K, sms, out)
        return {"swap": out[0], "BN": out[1], "splits": out[2], "workspace": int(need)}

    return f


def test_few_tokens_put_the_weight_on_the_lanes_and_split_k(plan):
    for M in (1, 8, 64, 65, 128):
        p = plan(M, 6144, 4096)
        assert p["swap"] == 1 and p["BN"] in (16, 32, 64, 128) and M <= p["BN"] < 2 * max(M, 16)
        assert p["splits"] == 4 and p["workspace"] == 4 * M * 6144 * 4      # 48 tiles x 4 = 192 CTAs in one wave
    assert plan(8, 4096, 4096)["splits"] == 8                               # 32 tiles x 8 = 256
    assert plan(8, 4096, 12288)["splits"] == 8
    assert plan(8, 24576, 4096)["splits"] == 3                              # 192 tiles: three splits fill 576 of 592 slots
    assert plan(8, 151936, 4096)["splits"] == 1                             # many waves: no split, no workspace
    assert plan(8, 151936, 4096)["workspace"] == 0


def test_many_tokens_are_left_whole_and_a_few_hundred_are_split_when_it_pays(plan):
    for N, K in [(6144, 4096), (4096, 4096), (24576, 4096), (4096, 12288)]:
        p = plan(2048, N, K)
        assert p["swap"] == 0 and p["BN"] == 256 and p["splits"] == 1
    assert plan(129, 4096, 12288)["swap"] == 0
    assert plan(160, 4096, 12288)["splits"] > 1      # 64 tiles on 148 SMs, 192 k-blocks each
    assert plan(160, 4096, 4096)["splits"] > 1
    assert plan(256, 6144, 4096)["splits"] == 1      # 48 tiles: the partial sums would cost what the split saves
    assert plan(512, 24576, 4096)["splits"] == 1


def test_without_room_for_a_cluster_products_stay_with_the_single_cta_kernel():
    """CTA pairs are planned for the clusters that the GPU holds: none of them, no pairs, and the plan is the single kernel's."""
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc to build the kernel library with")
    from zinfer_b200 import ops

    def f(M, N, K, pairs):
        out = (ctypes.c_int * 4)()
        ops.lib().zi_gemm_tcgen05_plan_for(M, N, K, 148, pairs, out)
        return tuple(out)

    for M, N, K in [(300, 4096, 12288), (536, 4096, 12288), (2048, 24576, 4096)]:
        assert f(M, N, K, 74)[3] == 1
        swap, BN, splits, pair = f(M, N, K, 0)
        assert pair == 0 and swap == 0 and BN in (128, 256) and splits >= 1
    assert f(2048, 24576, 4096, 20)[3] == 0        # 768 tiles in 39 rounds of 20 against 6 of 148 with twice the tiles each
    assert f(128, 24576, 4096, 74)[3] == 0


def test_a_product_with_a_fresh_weight_keeps_the_single_kernels_plan():
    """Where ``w`` is written earlier in the step the single-CTA kernel runs, by its own tile and splits and not by those of
    the pairs that the rule would have chosen."""
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc to build the kernel library with")
    from zinfer_b200 import ops

    for M, N, K in [(130, 4096, 4096), (300, 1024, 12288), (536, 4096, 12288), (257, 2050, 8200), (1024, 1280, 4160), (2048, 512, 2048)]:
        single, fresh = (ctypes.c_int * 4)(), (ctypes.c_int * 3)()
        ops.lib().zi_gemm_tcgen05_plan_for(M, N, K, 148, 0, single)
        need = ops.lib().zi_gemm_tcgen05_plan_fresh(M, N, K, 148, fresh)
        assert tuple(fresh) == tuple(single)[:3] and single[3] == 0
        assert need == (4 * fresh[2] * M * N if fresh[2] > 1 else 0)


@pytest.mark.parametrize("env,first", [(None, None), ("0", False), ("1", True)])
def test_the_switch_of_cta_pairs_gives_back_what_it_found(env, first):
    """Never, always, by the rule: the setting before, the environment's at first, comes back and is what the plans follow."""
    import os
    import subprocess
    import sys
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc to build the kernel library with")
    code = ("import ctypes\nfrom zinfer_b200 import ops\n"
            "def pairs(M, N, K):\n    p = (ctypes.c_int * 4)()\n    ops.lib().zi_gemm_tcgen05_plan_for(M, N, K, 148, 74, p)\n    return bool(p[3])\n"
            "shapes = [(2048, 24576, 4096), (384, 12288, 4096), (512, 256, 256)]\n"
            "found = [pairs(*s) for s in shapes]\n"
            f"assert ops.gemm_pair_kernel(False) is {first}\nassert not any(pairs(*s) for s in shapes)\n"
            "assert ops.gemm_pair_kernel(True) is False\nassert all(pairs(*s) for s in shapes[::2])\n"
            f"assert ops.gemm_pair_kernel({first}) is True\nassert [pairs(*s) for s in shapes] == found\n"
            "assert ops.gemm_pair_kernel(None) is " + str(first) + "\nassert pairs(*shapes[0])\nassert ops.gemm_pair_kernel(False) is None\n")
    env = {**{k: v for k, v in os.environ.items() if k != "ZINFER_B200_GEMM_PAIR"}, **({} if env is None else {"ZINFER_B200_GEMM_PAIR": env})}
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("M,N,K,splits", [
    # on pairs with so many splits, us on one B200 (single -> pair): 266 against 333, 127 against 144, 61 against 70 (with the
    # reader of the sums; 65 whole), 64 against 71, 42 against 45 (with the reader)
    (2048, 24576, 4096, 1), (1536, 4096, 12288, 1), (536, 4096, 12288, 3), (675, 4096, 12288, 1), (300, 4096, 12288, 2),
    # left to the single-CTA kernel (single, best of the pairs): 12.9 and 16.5 with the reader, 13.0 and 16.4, 11.9 and 13.2, 5.1 and
    # 5.7, 5.2 and 5.7, 6.2 and 7.0, 17.3 and 18.4
    (129, 4096, 4096, 0), (129, 2048, 8448, 0), (1300, 3072, 1024, 0), (512, 256, 256, 0), (256, 256, 256, 0), (257, 512, 512, 0), (675, 5120, 2048, 0)])
def test_pairs_are_planned_where_they_measured_faster(M, N, K, splits):
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc to build the kernel library with")
    from zinfer_b200 import ops

    plan = (ctypes.c_int * 4)()
    ops.lib().zi_gemm_tcgen05_plan_for(M, N, K, 148, 74, plan)
    assert plan[3] == (splits > 0) and (not splits or plan[2] == splits)


def test_splits_never_leave_a_split_without_k_blocks(plan):
    for M in (1, 8, 64, 65, 128, 300):
        for N, K in [(128, 64), (256, 512), (1000, 264), (4096, 4096), (5120, 17408), (151936, 4096)]:
            p = plan(M, N, K)
            kb = -(-K // 64)
            assert 1 <= p["splits"] <= kb
            assert (p["workspace"] > 0) == (p["splits"] > 1)


def test_sampling_rows_share_clusters_by_the_number_of_rows():
    if shutil.which("nvcc") is None:
        pytest.skip("no nvcc to build the kernel library with")
    from zinfer_b200 import ops

    f = ops.lib().zi_sample_ctas_per_row
    assert [f(r, 148) for r in (1, 8, 18, 19, 37, 38, 64, 74, 75, 256)] == [8, 8, 8, 4, 4, 2, 2, 2, 1, 1]
    assert f(1, 4) == 4 and f(5, 4) == 1
