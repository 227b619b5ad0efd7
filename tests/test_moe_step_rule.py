"""Which steps of a few tokens read every choice's weights for its token alone: by the choices against the distinct experts they can name."""
import pytest


@pytest.mark.parametrize("M,width,ff,experts,top,takes", [
    (1, 2048, 1024, 32, 4, True), (8, 2048, 1024, 32, 4, True), (8, 2048, 1024, 64, 8, True), (9, 2048, 1024, 32, 4, False),
    (6, 4096, 1024, 16, 4, True), (8, 4096, 1024, 16, 4, False), (8, 4096, 1024, 32, 4, True), (5, 4096, 1024, 64, 8, True), (6, 4096, 1024, 64, 8, False),
    (6, 2048, 2048, 16, 4, True), (8, 2048, 2048, 16, 4, False), (8, 2048, 2048, 32, 4, True), (8, 2048, 2048, 64, 8, False),
    (4, 4096, 2048, 16, 4, True), (4, 4096, 2048, 2, 1, True), (5, 4096, 2048, 2, 1, False), (8, 64, 32, 2, 2, True), (2, 60, 32, 4, 2, False)])
def test_rule(M, width, ff, experts, top, takes):
    from lit_llama.moe import step_pays

    assert step_pays(M, width, ff, 0, experts, top, 2) == takes
