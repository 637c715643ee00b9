"""Which evaluation a prompt of multi-head latent attention takes."""
import pytest

from fastllm_b200.ops import latent as LA


@pytest.mark.parametrize("H,n,keys,n_req,want", [
    # us: absorbed, expanded, folded
    (16, 17, 32785, 1, "absorbed"),        # 239 1047 333
    (16, 64, 32832, 1, "folded"),          # 746 1058 462
    (16, 200, 32968, 1, "folded"),         # 2217 1394 796
    (16, 1000, 33768, 1, "expanded"),      # 7749 1370 3030
    (16, 32, 4128, 1, "absorbed"),         # 81 166 184
    (16, 400, 4496, 1, "expanded"),        # 531 206 335
    (16, 64, 4160, 8, "expanded"),         # 722 342 1054
    (128, 8, 4104, 1, "absorbed"),         # 97 310 186
    (128, 32, 32800, 1, "folded"),         # 1418 2093 903
    (128, 256, 33024, 1, "expanded"),      # 9742 2493 5687
    (128, 1000, 1000, 1, "expanded"),      # 1376 220 1717
    (16, 2000, 2000, 2, "expanded")])
def test_choice_of_the_form(H, n, keys, n_req, want, monkeypatch):
    monkeypatch.setattr(LA, "EXPAND_BYTES", 1 << 40)          # (measured without slices)
    la = LA.LatentWeights()
    la.heads, la.dim, la.vdim, la.rank, la.lv, la.rot, la.rd, la.ld = H, 128, 128, 512, 512, 64, 64, 576
    assert LA.prompt_form(la, n, keys, n_req) == want


def test_latents_beyond_the_decode_kernel_are_not_absorbed():
    la = LA.LatentWeights()
    la.heads, la.dim, la.vdim, la.rank, la.lv, la.rot, la.rd, la.ld = 16, 128, 128, 1024, 1024, 64, 64, 1088
    assert LA.prompt_form(la, 4, 32000) == "folded" and LA.prompt_form(la, 4000, 4000) == "expanded"
