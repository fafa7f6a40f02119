"""Which form of the whole-step kernel serves a scene: the rule on sizes, and that a form which the
device refuses leaves the scene to the next one that serves it (host code, compiled here)."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include "pbf_small_form.h"
int main() {
  unsigned long long n, cells, sms;
  unsigned refused;  // bit f: the device refuses form f
  while (std::scanf("%llu %llu %llu %u", &n, &cells, &sms, &refused) == 4) {
    unsigned asked = 0;
    const int form = pbf::small_form_for(n, cells, sms, [&](int f) {
      asked |= 1u << f;
      return !(refused >> f & 1u);
    });
    std::printf("%d %u\n", form, asked);
  }
}
"""


@pytest.fixture(scope="module")
def form_of(tmp_path_factory):
    d = tmp_path_factory.mktemp("form")
    (d / "f.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(ROOT / "fluid_gb300" / "csrc"), "-o", str(d / "f"),
                    str(d / "f.cpp")], check=True)

    def run(rows):
        text = "\n".join(" ".join(str(x) for x in r) for r in rows)
        out = subprocess.run([str(d / "f")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(int(x) for x in ln.split()) for ln in out.splitlines()]
    return run


def test_sizes(form_of):
    rows = [(n, 1000, 152, 0) for n in (0, 1, 1024, 1025, 9728, 9729, 19456, 19457, 38912, 38913)]
    assert [f for f, _ in form_of(rows)] == [0, 1, 1, 2, 2, 3, 3, 4, 4, 0]
    # cells: 16 tiles of 1,024 for a cluster, a tile a block at most over the grid
    rows = [(500, c, 152, 0) for c in (16384, 16385, 304 * 1024, 304 * 1024 + 1)]
    assert [f for f, _ in form_of(rows)] == [1, 2, 2, 0]


def test_a_refused_form_leaves_the_scene_to_the_next(form_of):
    assert form_of([(500, 1000, 152, 1 << 1)])[0][0] == 2       # no clusters of 16 blocks
    assert form_of([(500, 1000, 152, 0b110)])[0][0] == 3
    assert form_of([(500, 1000, 152, 0b11110)])[0][0] == 0      # none: the per-phase kernels
    assert form_of([(12000, 1000, 152, 1 << 3)])[0] == (4, 0b11000)
    assert form_of([(500, 1000, 0, 0)])[0] == (0, 0)


def test_no_form_is_asked_in_vain(form_of):
    rng = np.random.default_rng(0)
    rows = [(int(10 ** rng.uniform(0, 5)), int(10 ** rng.uniform(1, 6)), int(rng.integers(1, 200)), 2 * int(rng.integers(16)))
            for _ in range(500)]
    for (n, cells, sms, refused), (form, asked) in zip(rows, form_of(rows)):
        per_block, room = (0, 64, 32, 128, 256), (0, 16, 2 * sms, sms, sms)
        serve = [f for f in range(1, 5) if -(-n // per_block[f]) <= room[f] and -(-cells // 1024) <= room[f]]
        taken = [f for f in serve if not refused >> f & 1]
        assert form == (taken[0] if taken else 0)
        assert asked == sum(1 << f for f in serve if not taken or f <= taken[0])


@pytest.mark.gpu
def test_forms_of_handles():
    import torch

    from fluid_gb300 import pbf, scenes

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ends = {1: (1, 1024), 2: (1025, 64 * sms), 3: (64 * sms + 1, 128 * sms), 4: (128 * sms + 1, 256 * sms),
            0: (256 * sms + 1,)}
    prm = scenes.physical_params(0.1, 0.05, max_neighbors=1024, iters=0)
    for form, counts in ends.items():
        for n in counts:
            p = np.random.default_rng(n).uniform(0, 1, (n, 3))
            with pbf.Simulator(p, np.zeros_like(p), prm) as sim:
                assert sim.step_form == form
                sim.set_collider_spheres([[0.5, 0.5, 0.5, 0.1]])
                assert sim.step_form == 0
                sim.set_collider_spheres(None)
                assert sim.step_form == form


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 500, 700, 1024, 1025, 3000, 9727, 9729, 12000, 19455, 19457, 38911])
def test_the_scenes_of_the_bit_comparison_take_the_whole_step_kernel(n):
    import torch

    from fluid_gb300 import pbf, scenes
    from tests.test_gpu_small_step import _state

    pos, vel, h = _state(n, seed=n)
    fits = n <= 256 * torch.cuda.get_device_properties(0).multi_processor_count
    with pbf.Simulator(pos, vel, scenes.physical_params(h, h / 2, max_neighbors=256)) as sim:
        assert (sim.step_form > 0) == fits
