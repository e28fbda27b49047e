"""The stage kernels (raygen, closest hit, shading with the emitter search)
against the CPU oracle.  Waves of up to 2 Mi paths run whole paths in one
kernel, so the comparisons of other files with the oracle reach the stages only
through their equality with it; here the same comparisons run with stage
timing, which keeps every wave in the stages."""
import pytest

import lisa_gb300 as L
import test_gpu_emitter_search as search
import test_gpu_physical as physical
import test_gpu_render as render

pytestmark = pytest.mark.gpu


@pytest.fixture
def stages(monkeypatch):
    """Renderers made in the test run stage by stage."""
    made = []

    class Staged(L.Renderer):
        def __init__(self, params, options=None, **kw):
            assert options is None
            super().__init__(params, **{**kw, "stage_timing": 1})

        def render(self, *a, **kw):
            st = super().render(*a, **kw)
            made.append(st.launches_nee)
            return st

    monkeypatch.setattr(L, "Renderer", Staged)
    yield
    assert made and min(made) > 0  # not k_paths


@pytest.mark.parametrize("light", ["point", "around", "far", "wall", "none"])
@pytest.mark.parametrize("width,height,spp", [(1, 1, 1), (33, 1, 1), (24, 17, 4), (160, 120, 8)])
def test_candidate_tries(gpu, oracle, stages, light, width, height, spp):
    search.test_candidate_tries_give_the_oracles_paths(gpu, oracle, light, width, height, spp)


def test_full_size_frame_band(gpu, oracle, stages):
    render.test_full_size_frame_band_path_by_path(gpu, oracle, "compat")


def test_full_size_soup_band(gpu, oracle, stages):
    render.test_full_size_soup_band_path_by_path(gpu, oracle)


def test_cornell_box(gpu, oracle, stages):
    render.test_path_by_path_cornell_box(gpu, oracle)


def test_hard_indirect(gpu, oracle, stages):
    render.test_path_by_path_hard_indirect(gpu, oracle)


def test_reference_stream(gpu, oracle, stages):
    render.test_path_by_path_reference_stream(gpu, oracle)


def test_many_materials(gpu, oracle, stages):
    render.test_path_by_path_sphere_soup_many_materials(gpu, oracle)


@pytest.mark.parametrize("focal", [0.0, 1.2])
def test_thin_lens(gpu, oracle, stages, focal):
    render.test_thin_lens_path_by_path(gpu, oracle, focal)


def test_physical_cornell_box(gpu, oracle, stages):
    physical.test_path_by_path_cornell_box(gpu, oracle)


def test_physical_icosphere(gpu, oracle, stages):
    physical.test_path_by_path_icosphere(gpu, oracle)


@pytest.mark.parametrize("name", [m for mark in render.test_matches_reference_shader_fixture.pytestmark
                                  if mark.name == "parametrize" for m in mark.args[1]])
def test_reference_shader_fixture(gpu, stages, tmp_path, name):
    render.test_matches_reference_shader_fixture(gpu, tmp_path, name)
