"""Models of every architecture in float32 at widths whose products run on tensor cores (weights of 2^20 numbers): a
product of up to 32 rows leaves its slices of K to the kernel behind it, whichever that is in the layer, and every logit
has the bits that it has where they are added first."""
import pytest
import torch

import brolm_b200 as bb
from brolm_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
W, H, D = 1024, 8, 128
EMBED = dict(architecture="", vocab=300, width=W, norm=dict(eps=1e-5))
SCALE = D ** -0.5
DECAY = [1.0 - 2.0 ** (-3.0 - h / 2) for h in range(H)]
ROT = dict(base=10000.0, dims=64, scaling=dict(factor=8.0, original=1024, fast=32.0, slow=1.0))
DENSE = dict(kind="dense", ff=2048)


def banevik():
    lat = dict(heads=H, dim=64, rot_dim=64, vdim=D, kv_rank=64, scale=SCALE, rot=dict(base=10000.0, dims=64), mask=dict(size=16))
    moe = dict(kind="moe", expert=dict(ff=1024), router=dict(experts=4, top=2))
    layers = [dict(type="latent_attention", mixer=lat, mlp=moe), dict(type="latent_attention", mixer=lat, mlp=moe)]
    return bb.BanevikConfig.from_dict(dict(EMBED, architecture="Banevik", layers=layers))


def neburax():
    moe = dict(kind="moe", expert=dict(ff=1024), router=dict(experts=4, top=2, identity=1), shared=dict(ff=1024))
    ssm = dict(heads=8, vdim=128, state=32, groups=2, norm_groups=2, conv=4)
    pair = dict(left=dict(heads=H, kv_heads=2, dim=D, vdim=D, scale=SCALE, mask=dict(size=16)),
                right=dict(width=W, blocks=4, conv=4), left_scale=1.0, right_scale=0.5)
    layers = [dict(type="mamba2", mixer=ssm, mlp=DENSE), dict(type="parallel", mixer=pair, mlp=moe)]
    return bb.NeburaxConfig.from_dict(dict(EMBED, architecture="Neburax", layers=layers))


def kedasun():
    mlp = dict(kind="dense", ff=2048, limit=7.0)
    rotary = dict(type="attention", mlp=mlp, mixer=dict(heads=H, kv_heads=2, dim=D, vdim=D, scale=SCALE, v_mix=True,
                                                        rot=dict(base=10000.0, dims=64)))
    windowed = dict(type="attention_2", mlp=mlp, mixer=dict(heads=H, kv_heads=2, dim=D, vdim=D, scale=SCALE, conv=4, v_mix=True,
                                                            mask=dict(size=16, keep_first=4)))
    return bb.KedasunConfig.from_dict(dict(EMBED, architecture="Kedasun", layers=[rotary, windowed], embedding=dict(scale=1.0),
                                           norm=dict(eps=1e-5, groups=4)))


def ritirax():
    moe = dict(kind="moe", expert=dict(ff=1024), shared=dict(ff=1024),
               router=dict(experts=8, top=2, scale=2.0, groups=dict(count=4, keep=2)))
    light = dict(heads=H, dim=D, vdim=D, decay=DECAY)
    attn = dict(heads=H, kv_heads=2, dim=D, vdim=D, scale=SCALE, softcap=30.0, bias_max=128, bias_rows=32)
    lat = dict(heads=H, dim=64, rot_dim=64, vdim=D, kv_rank=64, scale=SCALE, rot=ROT)
    layers = [dict(type="lightning", mixer=light, mlp=DENSE), dict(type="attention", mixer=attn, mlp=moe),
              dict(type="latent_attention", mixer=lat, mlp=moe)]
    return bb.RitiraxConfig.from_dict(dict(EMBED, architecture="Ritirax", layers=layers, embedding=dict(scale=W ** 0.5)))


def relulix():
    moe = dict(kind="moe", expert=dict(ff=1024, limit=7.0), router=dict(experts=4, top=2))
    ret = dict(heads=H, dim=D, vdim=D, decay=DECAY, rot=dict(base=10000.0, dims=D))
    attn = dict(heads=H, kv_heads=2, dim=D, vdim=D, scale=SCALE, softcap=30.0, mask=dict(size=16), rot=ROT)
    layers = [dict(type="retention", mixer=ret, mlp=moe), dict(type="attention", mixer=attn, mlp=moe)]
    return bb.RelulixConfig.from_dict(dict(EMBED, architecture="Relulix", layers=layers, embedding=dict(scale=W ** 0.5)))


def papusun():
    left = dict(heads=H, kv_heads=2, dim=D, vdim=D, scale=SCALE, softcap=30.0,
                rot=dict(base=10000.0, dims=D, scaling=dict(factor=8.0, low=1.0, high=4.0, original=1024)))
    pair = dict(left=left, right=dict(heads=H, kv_heads=H, dim=D, vdim=D, conv=4), left_scale=1.0, right_scale=0.5)
    lat = dict(heads=H, dim=64, rot_dim=64, vdim=D, q_rank=1024, kv_rank=64, scale=SCALE, mask=dict(size=16),
               rot=dict(base=10000.0, dims=64))
    layers = [dict(type="parallel", mixer=pair, mlp=DENSE), dict(type="latent_attention", mixer=lat, mlp=DENSE)]
    return bb.PapusunConfig.from_dict(dict(EMBED, architecture="Papusun", layers=layers, token_side=dict(dim=1024), logit_scale=0.25))


@pytest.mark.parametrize("config", [banevik, neburax, kedasun, ritirax, relulix, papusun], ids=lambda f: f.__name__)
def test_slices_left_to_the_kernel_behind_give_the_bits_of_those_added_first(monkeypatch, config):
    model = bb.Model(config(), dtype="float32", device=DEV).init_random(seed=4, on_device=True)
    g = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, 300, (n,), generator=g).tolist() for n in (19, 3, 8)]
    follow = torch.randint(0, 300, (4, 3), generator=g).tolist()
    sliced = []
    real = kernels.linear_f32_slices_into
    monkeypatch.setattr(kernels, "linear_f32_slices_into", lambda *a, **kw: sliced.append(1) or real(*a, **kw))

    def run():
        eng = bb.Engine(model, max_tokens=512, max_slots=3)
        slots = eng.open(3)
        rows = [eng.step(slots, prompts, want=[list(range(len(p))) for p in prompts]).clone()]
        rows += [eng.step(slots, [[t] for t in toks]).clone() for toks in follow]
        eng.close(slots)
        return torch.cat(rows)
    left = run()
    assert len(sliced) >= 4 and bool(left.isfinite().all())
    monkeypatch.setattr(kernels, "linear_f32_parts", lambda x, w: 1)
    n = len(sliced)
    assert torch.equal(run(), left) and len(sliced) == n
    monkeypatch.setattr(kernels, "linear_f32_tc_ok", lambda w: False)          # fmas: another rounding, no more
    assert float((run() - left).abs().max()) <= 1e-3 * float(left.abs().max())
