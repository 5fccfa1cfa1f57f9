"""Terms of a bounce that shading leaves out when a material lacks the lobe (clearcoat, sheen and tint,
absorption): path radiance equals the oracle's bit for bit with every such parameter at +0, -0 and
beyond, for rough, smooth, metallic and transmissive surfaces."""
import numpy as np
import pytest

import lavaframe_gb300 as lf
import oracle

pytestmark = pytest.mark.gpu


def material(albedo, specular, metallic, roughness, tint, sheen, sheen_tint, coat, coat_rough, trans, extinction):
    m = np.zeros(28, np.float32)
    m[0:3], m[3] = albedo, specular
    m[8], m[9], m[10], m[11] = metallic, roughness, 0.2, tint
    m[12], m[13], m[14], m[15] = sheen, sheen_tint, coat, coat_rough
    m[16], m[17], m[18] = trans, 1.45, 0.5
    m[20:23] = extinction
    m[24:28] = -1.0
    return m


ZEROS = [0.0, -0.0, 0.3]


@pytest.mark.parametrize("tint", ZEROS)
@pytest.mark.parametrize("sheen", ZEROS)
@pytest.mark.parametrize("coat", ZEROS)
@pytest.mark.parametrize("kind", ["rough", "mirror", "metal", "glass", "black", "negative"])
def test_bounces_equal_the_oracle(tint, sheen, coat, kind):
    metallic, rough, trans, albedo = {"rough": (0.0, 0.9, 0.0, (0.7, 0.5, 0.2)), "mirror": (0.1, 0.0, 0.0, (0.9, 0.9, 0.9)),
                                      "metal": (1.0, 0.2, 0.0, (0.9, 0.6, 0.1)), "glass": (0.0, 0.05, 1.0, (1, 1, 1)),
                                      "black": (0.0, 0.5, 0.0, (0, -0.0, 0)),
                                      "negative": (0.0, 0.5, 0.0, (0.2, -0.1, 0.1))}[kind]
    s = lf.HostScene()
    a = lf.HostScene().gen_icospheres(2, 2, 3, 40, 21).build().arrays()   # an environment of odd size
    r = np.random.default_rng(1)
    for k, extinction in enumerate(((1, 1, 1), (0.3, 0.6, 1.0))):
        v = np.zeros((60, 4), np.float32)
        v[:, :3] = r.standard_normal((60, 3)) + [1.5 * k, 0, 0]
        v[:, 3] = r.random(60)
        n = np.zeros((60, 4), np.float32)
        n[:, :3] = r.standard_normal((60, 3))
        n[:, :3] /= np.linalg.norm(n[:, :3], axis=1, keepdims=True)
        mid = s.add_mesh(v, n)
        mat = s.add_material(material(albedo, 0.5, metallic, rough, tint, sheen, 0.4, coat, 0.7, trans, extinction))
        s.add_instance(mid, np.eye(4, dtype=np.float32).ravel(), mat)
    light = np.zeros(15, np.float32)
    light[0:3], light[3:6], light[6:9], light[9:12], light[13] = (-1, 4, -1), (9, 8, 7), (2, 0, 0), (0, 0, 2), 4.0
    s.add_light(light)
    s.add_hdr(a["env_rgb"])
    s.set_camera([0.5, 0.5, 5.0], [0.5, 0.0, 0.0], 50.0)
    s.build()
    p = s.render_params()
    p.width, p.height, p.max_depth, p.use_env_map = 24, 16, 5, 1
    with lf.Context(0) as ctx:
        ds = ctx.upload(s)
        f = lf.Frame(ctx, ds, p)
        f.render(0, 4)
        got = f.paths(4)
        f.close()
        ds.close()
    _, want, _ = oracle.render(s.view(), p, 0, 4, want_paths=True)
    assert (want != 0).any()
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert same.all()
