"""The RGBA8 -> RGBA16F conversion, moved in pairs of texels and slices where the buffers' alignment allows: every
texel is half(b / 255), at resolutions whose slices and tiles leave remainders, aligned or not, mirrored or not."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [8, 16, 64])
@pytest.mark.parametrize("src_off,dst_off", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("mirrored", [False, True])
def test_every_texel_is_the_half_of_its_quotient(cuda, R, src_off, dst_off, mirrored):
    torch = cuda
    from vk_voxel_cone_tracing_gb300 import capi, clipmap
    n = (6 * (R + 2)) ** 2 * (R + 2)
    g = torch.Generator(device="cuda").manual_seed(R)
    src = torch.randint(-2 ** 31, 2 ** 31 - 1, (n + 2,), dtype=torch.int32, device="cuda", generator=g)[src_off:][:n]
    room = torch.full(((n + 2) * 4,), 7, dtype=torch.int16, device="cuda")
    dst = room[4 * dst_off:][:4 * n]
    tex = clipmap.RadianceTexture(R, capi.TEX_RGBA16F) if mirrored else None
    clipmap.to_rgba16f(src, R, out=dst, mirror=tex)
    want = (src.view(torch.uint8).float() / 255.0).half()
    assert torch.equal(dst.view(torch.float16), want)
    assert (room[:4 * dst_off] == 7).all() and (room[4 * (dst_off + n):] == 7).all()
    if tex is not None:
        back = tex.read(clipmap.new_atlas_rgba16f(R, src.device))
        torch.cuda.synchronize()
        assert torch.equal(back.view(-1).view(torch.float16), want)
        tex.close()
