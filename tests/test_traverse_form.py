"""The launch of a CWBVH traversal (obvhs_gb300/csrc/traverse_form.h, compiled
for the host): a form that a context has chosen is taken for calls of every
size; the default form gives each warp fewer rays in calls of few.  On the GPU:
equal hits in every form below, at and above the count where that begins, and
an autotuner call that large."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "obvhs_gb300", "csrc")
FORMS = ((128, 0), (64, 0), (256, 0), (64, 1), (128, 1))


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("tf") / "traverse_form_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", CSRC, os.path.join(HERE, "traverse_form_check.cpp"), "-o", exe],
                   check=True)

    def ask(cases):
        out = subprocess.run([exe, *(str(int(v)) for c in cases for v in c)], capture_output=True, text=True, check=True)
        return [tuple(int(v) for v in line.split()) for line in out.stdout.splitlines()]

    return ask


COUNTS = (1, 31, 1000, 1215, 1216, 1217, 19_455, 19_456, 19_457, 100_000, 2**32 - 1)


def test_a_chosen_form_is_taken_for_every_count(rule):
    for f, (block, smem) in enumerate(FORMS):
        for form, lanes in rule([(sms, n, block, smem) for sms in (1, 148, 152) for n in COUNTS]):
            assert form == f
            assert f == 0 or lanes == 32


def test_the_default_spreads_few_rays(rule):
    for sms in (1, 148, 152):
        cases = [(sms, n, 0, 0) for n in COUNTS]
        for (_, n, _, _), (form, lanes) in zip(cases, rule(cases)):
            assert form == 0
            # the fewest of 1, 2, ... 32 with at most two warps for each of four schedulers
            assert lanes == next((r for r in (1, 2, 4, 8, 16) if r * sms * 8 >= n), 32)


def test_no_such_form(rule):
    assert all(form == -1 for form, _ in rule([(152, 5, 32, 0), (152, 5, 256, 1), (152, 5, 0, 1), (152, 5, 100, 0)]))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 1000, 19_456, 19_457])
def test_hits_are_equal_in_every_form(n):
    import obvhs_gb300 as G
    from obvhs_gb300 import scenes as S
    from obvhs_gb300 import test_util as T
    from obvhs_gb300.params import BvhBuildParams

    rng = np.random.default_rng(n)
    d = T.uniform_sample_sphere(rng.random(n).astype(np.float32), rng.random(n).astype(np.float32))
    rays = T.make_rays(rng.uniform(-10, 10, size=(n, 3)).astype(np.float32), d, 0.0,
                       rng.uniform(0.5, 40, size=n).astype(np.float32))
    with G.Context() as ctx:
        cw = G.build_cwbvh_from_tris(S.scene2_tris(20_000), BvhBuildParams.medium_build(), ctx=ctx)
        ids, t = cw.ray_traverse(rays)
        miss = cw.ray_traverse_miss(rays)
        for block, smem in G.Context.TRAVERSAL_CONFIGS:
            ctx.set_traversal_config(block, smem)
            got_ids, got_t = cw.ray_traverse(rays)
            assert np.array_equal(got_ids, ids) and np.array_equal(got_t.view(np.uint32), t.view(np.uint32))
            assert np.array_equal(cw.ray_traverse_miss(rays), miss)
        cw.free()


@pytest.mark.gpu
def test_autotuner_above_the_few_ray_counts():
    import torch

    import obvhs_gb300 as G
    from obvhs_gb300 import autotune as A
    from obvhs_gb300 import scenes as S
    from obvhs_gb300 import test_util as T
    from obvhs_gb300.params import BvhBuildParams

    n = 16 * 8 * torch.cuda.get_device_properties(0).multi_processor_count + 1
    rng = np.random.default_rng(5)
    d = T.uniform_sample_sphere(rng.random(n).astype(np.float32), rng.random(n).astype(np.float32))
    rays = torch.from_numpy(T.make_rays(rng.uniform(-10, 10, size=(n, 3)).astype(np.float32), d, 0.0, np.inf)).cuda()
    with G.Context() as ctx:
        cw = G.build_cwbvh_from_tris(S.scene2_tris(20_000), BvhBuildParams.medium_build(), ctx=ctx)
        got = A.tune_traversal(lambda: cw.ray_traverse(rays), ctx, reps=1)
        assert (got["block"], got["smem_stack"]) in G.Context.TRAVERSAL_CONFIGS
        assert len(got["ms"]) == len(G.Context.TRAVERSAL_CONFIGS)
        cw.free()
