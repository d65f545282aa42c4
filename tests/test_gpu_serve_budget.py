"""A scene's build takes memory that the scene does not keep: the server charges it
while the build runs, so that the budget holds, and gives the charge back."""
import pytest

from rtgb import capi, scenes

pytestmark = pytest.mark.gpu

ARENA = 16 << 20
N = 200000          # triangles; a build's scratch is 18 B for each and more


@pytest.fixture(scope="module")
def mesh():
    return [scenes.soup(N, seed=71 + k) for k in range(3)]


@pytest.fixture(scope="module")
def one(ctx, mesh):
    """Bytes of the resident scene."""
    srv = capi.Server(ctx, budget=1 << 30, arena=ARENA, max_views=8, max_inflight=1)
    srv.add_scene(mesh[0])
    n = srv.stats().resident_bytes - ARENA
    srv.close()
    return n


def test_a_build_that_does_not_fit_is_rejected(ctx, mesh, one):
    srv = capi.Server(ctx, budget=ARENA + one + 10 * N, arena=ARENA, max_views=8, max_inflight=1)
    with pytest.raises(capi.RtError):
        srv.add_scene(mesh[0])
    _, inf = srv.result(srv.submit_upload(mesh[0]), raise_on_error=False)
    assert inf.status == -8
    assert srv.stats().resident_bytes == ARENA
    srv.close()


@pytest.mark.parametrize("submit", [False, True])
def test_the_charge_of_a_build_is_given_back(ctx, mesh, one, submit):
    """Room for two scenes and one build: the second build waits for the first,
    a third scene takes the place of one of them."""
    srv = capi.Server(ctx, budget=ARENA + 2 * one + 30 * N, arena=ARENA, max_views=8, max_inflight=1)
    if submit:
        tickets = [srv.submit_upload(m) for m in mesh[:2]]
        ids = [srv.result(t)[1].scene_id for t in tickets]
    else:
        ids = [srv.add_scene(m) for m in mesh[:2]]
    st = srv.stats()
    assert st.resident_scenes == 2 and st.evicted == 0 and st.rejected == 0
    assert st.resident_bytes == ARENA + 2 * one
    cam = scenes.camera((0, 0, -4), (0, 0, 0))
    for i in ids:
        assert srv.result(srv.submit_render(i, cam, 32, 32, 1), 32, 32)[1].status == 0
    assert srv.result(srv.submit_upload(mesh[2]))[1].status == 0
    st = srv.stats()
    assert st.resident_scenes == 2 and st.evicted == 1 and st.resident_bytes == ARENA + 2 * one
    srv.close()
