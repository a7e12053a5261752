"""The fused decode stack (one cooperative launch for 1..64 tokens) against the CPU path and against the
layer-by-layer launches it replaces: rel-RMSE <= 1e-5 for a single f32 layer, identical routing decisions, a
bf16 stack that follows the layer-by-layer stack to within rounding flips, and the bounded-wait give-up path."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
from gpu_util import dev, report
from kanjoos_b200 import synth

pytestmark = pytest.mark.gpu


def _banks(cfg, L, E, H, F):
    from kanjoos_b200.moe import ExpertBank
    banks, cpu = [], []
    for l in range(L):
        bank = synth.expert_bank(cfg, l, n_experts=E, hidden=H, ffn=F)
        wr, _ = synth.router_weight(cfg, l, n_experts=E, hidden=H)
        nb = synth.norm_weight(cfg, l, H)
        banks.append(ExpertBank.from_numpy(bank, wr, None, nb))
        cpu.append((bank, wr, nb))
    return banks, cpu


@pytest.mark.parametrize("T,E,H,F,k", [(1, 16, 512, 256, 4), (3, 16, 512, 256, 4), (4, 32, 1024, 512, 8),
                                      (1, 128, 2048, 768, 8), (2, 128, 2048, 768, 8), (8, 128, 2048, 768, 8),
                                      (17, 16, 512, 256, 4), (64, 128, 2048, 768, 8), (64, 8, 768, 256, 2)])
def test_single_layer_f32_against_cpu_path(T, E, H, F, k):
    from kanjoos_b200.moe import FusedMoeStack, MoeFfnLayer
    banks, cpu = _banks(801, 1, E, H, F)
    hx = synth.hidden_rows(801, T, H, layer=T)
    st = FusedMoeStack(banks, top_k=k, n_tokens=T, dtype=torch.float32, residual=False, taps=True)
    got = st.step(dev(hx)).cpu().numpy()
    st.status()
    bank, wr, nb = cpu[0]
    xn = ol.rmsnorm(hx, synth.bf16_bits_to_f32(nb), synth.RMS_EPS)
    want, _, _ = ol.moe(wr, bank, xn, k)
    assert report(got, want, f"fused stack, 1 layer, T={T}")["rel_rmse"] <= 1e-5
    # the same routing decisions (experts and weights) as the layer-by-layer launch
    layer = MoeFfnLayer(banks[0], top_k=k, max_tokens=T, residual=False)
    _, pe, pw = layer.decode(dev(hx), return_routing=True)
    assert torch.equal(pe, st.taps[0][0]) and torch.equal(pw.view(torch.int32), st.taps[0][1].view(torch.int32))
    st.close()


@pytest.mark.parametrize("T,E", [(16, 128), (17, 128), (32, 128), (33, 100), (48, 128), (61, 128), (33, 160)])
def test_routing_is_the_layer_launch_s_at_every_group_of_tokens(T, E):
    """The stack's plan selects one, two or four tokens per warp at a time (and one from 129 experts on): the same
    experts and the same bits of the weights as the layer launch, whose front kernel takes one."""
    from kanjoos_b200.moe import FusedMoeStack, MoeFfnLayer
    H, F, k = 512, 256, 8
    banks, _ = _banks(806, 1, E, H, F)
    x = dev(synth.hidden_rows(806, T, H))
    st = FusedMoeStack(banks, top_k=k, n_tokens=T, dtype=torch.float32, residual=False, taps=True)
    st.step(x)
    st.status()
    _, pe, pw = MoeFfnLayer(banks[0], top_k=k, max_tokens=T, residual=False).decode(x, return_routing=True)
    assert torch.equal(pe, st.taps[0][0]) and torch.equal(pw.view(torch.int32), st.taps[0][1].view(torch.int32))
    st.close()


@pytest.mark.parametrize("T", [1, 2, 9, 33])
def test_masked_experts(T):
    """Biases of -inf that leave three experts to a top-4: the fourth is a masked one with weight 0, so the layer launch and
    the stack (both kernels) give what top-3 gives, bit for bit; with every expert masked the rows pass through."""
    from kanjoos_b200.moe import FusedMoeStack, MoeFfnLayer
    E, H, F = 16, 512, 256
    banks, _ = _banks(811, 1, E, H, F)
    x = dev(synth.hidden_rows(811, T, H))
    for finite in ([2, 7, 15], []):
        bias = torch.full((E,), float("-inf"), device="cuda")
        bias[finite] = 0.0
        banks[0].router_bias = bias
        want = MoeFfnLayer(banks[0], top_k=3, max_tokens=T, residual=True).decode(x) if finite else x
        assert torch.equal(MoeFfnLayer(banks[0], top_k=4, max_tokens=T, residual=True).decode(x), want)
        stacks = [FusedMoeStack(banks, top_k=k, n_tokens=T, dtype=torch.float32, taps=True) for k in (3, 4)]
        got = [st.step(x).clone() for st in stacks]
        for st in stacks:
            st.status()
            assert ((st.taps[0][0] >= 0) & (st.taps[0][0] < E)).all()
            st.close()
        assert torch.equal(got[1], got[0] if finite else x)


def test_stack_follows_layer_by_layer_launches():
    from kanjoos_b200.moe import FusedMoeStack, MoeStack
    L, E, H, F, k, T = 6, 32, 1024, 512, 8, 2
    banks, cpu = _banks(802, L, E, H, F)
    x0 = synth.bf16_round(synth.hidden_rows(802, T, H) * 200.0)
    x = dev(x0).to(torch.bfloat16)
    ref = MoeStack(banks, top_k=k, max_tokens=T).step(x).float().cpu().numpy()
    st = FusedMoeStack(banks, top_k=k, n_tokens=T)
    got = st.step(x).float().cpu().numpy()
    st.status()
    again = st.step(x).float().cpu().numpy()      # a second launch: the barrier words start over
    st.status()
    assert np.array_equal(got, again)
    s = report(got, ref, "fused vs layer-by-layer, 6 layers, bf16 stream")
    assert s["rel_rmse"] <= 1e-2 and np.mean(got != ref) < 0.02   # only bf16 rounding flips apart
    cur = x0
    for bank, wr, nb in cpu:
        xn = ol.rmsnorm(cur, synth.bf16_bits_to_f32(nb), synth.RMS_EPS)
        mo, _, _ = ol.moe(wr, bank, xn, k)
        cur = synth.bf16_round(cur + mo)
    assert report(got, cur, "fused vs CPU path, 6 layers")["rel_rmse"] <= 1e-2
    st.close()


@pytest.mark.parametrize("T", [8, 64])
def test_stack_follows_layer_by_layer_launches_larger_batches(T):
    from kanjoos_b200.moe import FusedMoeStack, MoeStack
    L, E, H, F, k = 4, 32, 1024, 512, 8
    banks, _ = _banks(804, L, E, H, F)
    x0 = synth.bf16_round(synth.hidden_rows(804, T, H) * 200.0)
    x = dev(x0).to(torch.bfloat16)
    ref = MoeStack(banks, top_k=k, max_tokens=T).step(x).float().cpu().numpy()
    st = FusedMoeStack(banks, top_k=k, n_tokens=T)
    got = st.step(x).float().cpu().numpy()
    st.status()
    s = report(got, ref, f"fused vs layer-by-layer, {L} layers, bf16 stream, T={T}")
    assert s["rel_rmse"] <= 1e-2 and np.mean(got != ref) < 0.02
    st.close()


def _q6k_down(cfg, E, H, F):
    rng = np.random.Generator(np.random.Philox(cfg))
    W6 = rng.integers(0, 256, size=(E, H, F // 256, 210), dtype=np.uint8)
    W6[..., 208:210] = (np.abs(rng.standard_normal((E, H, F // 256, 1))) * 0.01).astype(np.float16).view(np.uint8)
    return W6


@pytest.mark.parametrize("T", [1, 3, 8, 37, 64])
def test_mixed_format_stack_q6k_down_follows_the_layer_launches(T):
    """A stack as Q4_K_M files hold it: the down matrices of every other layer are Q6_K. The whole-stack launch
    takes them through its own down phase; the layer-by-layer launches (whose Q6_K projection is checked against
    the CPU decoder) are the comparison, f32 stream so that nothing but summation order may differ."""
    from kanjoos_b200.moe import ExpertBank, FusedMoeStack, MoeStack
    L, E, H, F, k = 4, 16, 512, 512, 4
    banks = []
    for l in range(L):
        bank = synth.expert_bank(806, l, n_experts=E, hidden=H, ffn=F)
        if l % 2 == 1:
            bank = dict(bank, down=_q6k_down(806 + l, E, H, F))
        wr, _ = synth.router_weight(806, l, n_experts=E, hidden=H)
        banks.append(ExpertBank.from_numpy(bank, wr, None, synth.norm_weight(806, l, H)))
    x = dev(synth.hidden_rows(806, T, H))
    ref = MoeStack(banks, top_k=k, max_tokens=T).step(x).cpu().numpy()
    st = FusedMoeStack(banks, top_k=k, n_tokens=T, dtype=torch.float32)
    got = st.step(x).cpu().numpy()
    st.status()
    s = report(got, ref, f"mixed-format stack (Q6_K down in layers 1 and 3), T={T}, fused vs layer launches")
    assert s["unwritten"] == 0 and s["rel_rmse"] <= 1e-5
    st.close()


@pytest.mark.parametrize("F,T", [(256, 1), (256, 20), (768, 5), (768, 33), (1024, 3), (1024, 20)])
def test_q6k_down_phase_follows_the_layer_launch_at_every_row_length(F, T):
    """One Q6_K layer: tiles of one, three and four superblocks (four leave room for twelve warps' tiles, not sixteen),
    experts of one and of several jobs of four tokens, against the layer launch's own Q6_K projection."""
    from kanjoos_b200.moe import ExpertBank, FusedMoeStack, MoeFfnLayer
    E, H, k = 12, 512, 4
    bank = dict(synth.expert_bank(808, 0, n_experts=E, hidden=H, ffn=F), down=_q6k_down(808, E, H, F))
    wr, _ = synth.router_weight(808, 0, n_experts=E, hidden=H)
    b = ExpertBank.from_numpy(bank, wr, None, synth.norm_weight(808, 0, H))
    x = dev(synth.hidden_rows(808, T, H))
    want = MoeFfnLayer(b, top_k=k, max_tokens=T, residual=True).decode(x).cpu().numpy()
    st = FusedMoeStack([b], top_k=k, n_tokens=T, dtype=torch.float32)
    got = st.step(x).cpu().numpy()
    st.status()
    st.close()
    assert report(got, want, f"Q6_K down phase, ffn {F}, T={T}")["rel_rmse"] <= 1e-5


@pytest.mark.parametrize("F,T,E", [(768, 8, 32), (768, 64, 16), (1024, 8, 16), (1024, 64, 32)])
def test_q6k_down_phase_with_more_tiles_than_warps(F, T, E):
    """At hidden 2048 a CTA has more tiles than warps that take them (128 tiles a job, 16 at ffn 768 and 12 at ffn 1024), so a
    warp copies tile after tile into its one buffer; a Q4_K layer between two Q6_K layers hands the barriers' phases and the
    ring area over both ways. Against the layer launches, f32 stream: nothing but summation order may differ."""
    from kanjoos_b200.moe import ExpertBank, FusedMoeStack, MoeStack
    L, H, k = 3, 2048, 8
    banks = []
    for l in range(L):
        bank = synth.expert_bank(813, l, n_experts=E, hidden=H, ffn=F)
        if l != 1:
            bank = dict(bank, down=_q6k_down(813 + l, E, H, F))
        wr, _ = synth.router_weight(813, l, n_experts=E, hidden=H)
        banks.append(ExpertBank.from_numpy(bank, wr, None, synth.norm_weight(813, l, H)))
    x = dev(synth.hidden_rows(813, T, H))
    ref = MoeStack(banks, top_k=k, max_tokens=T).step(x).cpu().numpy()
    st = FusedMoeStack(banks, top_k=k, n_tokens=T, dtype=torch.float32, taps=True)
    got = st.step(x).cpu().numpy()
    st.status()
    for l in (0, 2):
        jobs = int(((torch.bincount(st.taps[l][0].flatten().long(), minlength=E) + 3) // 4).sum())
        assert jobs * (H // 16) > (16 if F == 768 else 12) * torch.cuda.get_device_properties(0).multi_processor_count, jobs
    assert np.array_equal(got, st.step(x).cpu().numpy())
    st.status()
    st.close()
    s = report(got, ref, f"Q6_K down phase of several tiles a warp, ffn {F}, T={T}")
    assert s["unwritten"] == 0 and s["rel_rmse"] <= 1e-5


@pytest.mark.parametrize("B", [1, 8, 64])
def test_config4_full_size_stack_checked_layers(B):
    """Config 4: the 48-layer resident stack at full size (about 15 GiB of random-init Q4_K experts), f32 residual
    stream. Layers 0, 1, 23 and 47 are checked against the CPU path fed with the GPU's own layer input: tokens
    whose routed expert sets agree (all but near-ties) within 1e-5, and nearly all tokens must agree."""
    from kanjoos_b200.moe import ExpertBank, FusedMoeStack
    L, k = 48, 8
    free, _ = torch.cuda.mem_get_info()
    if free < 20 * 2**30:
        pytest.skip("needs 20 GiB of free device memory")
    banks = [ExpertBank.random(seed=4000 + l) for l in range(L)]
    g = torch.Generator(device="cuda")
    g.manual_seed(B)
    x = torch.randn((B, synth.HIDDEN), device="cuda", generator=g)
    st = FusedMoeStack(banks, top_k=k, n_tokens=B, dtype=torch.float32, taps=True, keep_outputs=True)
    st.step(x)
    st.status()
    for l in (0, 1, 23, 47):
        b = banks[l]
        bank = {"gate": b.gate.cpu().numpy(), "up": b.up.cpu().numpy(), "down": b.down.cpu().numpy()}
        wr = b.router.view(torch.int16).cpu().numpy().view(np.uint16)
        nw = b.norm_w.view(torch.int16).cpu().numpy().view(np.uint16)
        xin = (x if l == 0 else st.outs[l - 1]).cpu().numpy()
        xn = ol.rmsnorm(xin, synth.bf16_bits_to_f32(nw), b.rms_eps)
        mo, ch_cpu, _ = ol.moe(wr, bank, xn, k)
        want = xin + mo
        got = st.outs[l].cpu().numpy()
        ch_gpu = st.taps[l][0].cpu().numpy().reshape(B, k)
        same = np.array([set(ch_gpu[t]) == set(ch_cpu[t]) for t in range(B)])
        assert same.mean() >= 0.9, f"layer {l}: routed sets differ for {int((~same).sum())} of {B} tokens"
        s = report(got[same], want[same], f"48-layer stack, batch {B}, layer {l} ({int(same.sum())} tokens)")
        assert s["rel_rmse"] <= 1e-5
    st.close()


def test_bounded_wait_gives_up_and_the_stack_recovers():
    """A grid barrier whose target cannot be reached runs into its limit: the launch returns, status() reports
    KNJ_E_TIMEOUT (-5), nothing traps, and the next normal launch on the same stack is right again."""
    from kanjoos_b200 import _lib
    from kanjoos_b200.moe import FusedMoeStack
    banks, cpu = _banks(805, 2, 16, 512, 256)
    hx = synth.hidden_rows(805, 2, 512)
    st = FusedMoeStack(banks, top_k=4, n_tokens=2, dtype=torch.float32, residual=False)
    want = st.step(dev(hx)).cpu().numpy().copy()
    st.status()
    st.set_wait(wait_cycles=2_000_000, stall_first_barrier=1)   # about a millisecond, then every CTA returns
    st.step(dev(hx))
    with pytest.raises(_lib.KnjError) as ei:
        st.status()
    assert ei.value.code == -5
    st.set_wait(0, 0)
    got = st.step(dev(hx)).cpu().numpy()
    st.status()
    assert np.array_equal(got, want)
    st.close()


@pytest.mark.parametrize("down", ["q4k", "q6k"])
@pytest.mark.parametrize("warp", [0, 2, 9])
def test_a_copy_that_does_not_land_is_reported_whichever_warp_waits(down, warp):
    """The first weight copies of one warp of CTA 0 never count as landed: status() reports KNJ_E_TIMEOUT although the CTA's
    other warps land theirs, and the next normal launch is right again. Jobs of 32 gate+up tiles and 112 down tiles, 14 to
    41 of them over 148 CTAs: warps 0 and 2 already wait in the gate+up phase (3 to 8 tiles a CTA), warp 9 in the down
    phase alone (10 and more)."""
    from kanjoos_b200 import _lib
    from kanjoos_b200.moe import ExpertBank, FusedMoeStack
    E, H, F, T, k = 16, 1792, 256, 8, 8
    bank = synth.expert_bank(812, 0, n_experts=E, hidden=H, ffn=F)
    if down == "q6k":
        bank = dict(bank, down=_q6k_down(812, E, H, F))
    wr, _ = synth.router_weight(812, 0, n_experts=E, hidden=H)
    b = ExpertBank.from_numpy(bank, wr, None, synth.norm_weight(812, 0, H))
    x = dev(synth.hidden_rows(812, T, H))
    st = FusedMoeStack([b], top_k=k, n_tokens=T, dtype=torch.float32, taps=True)
    want = st.step(x).clone()
    st.status()
    jobs = int(((torch.bincount(st.taps[0][0].long(), minlength=E) + 3) // 4).sum())
    assert 14 <= jobs <= 41
    st.set_wait(wait_cycles=2_000_000)   # about a millisecond
    _lib.check(_lib.lib().knj_moe_stack_test_stall_copy(st._h, warp))
    st.step(x)
    with pytest.raises(_lib.KnjError) as ei:
        st.status()
    assert ei.value.code == -5
    st.set_wait(0)
    _lib.check(_lib.lib().knj_moe_stack_test_stall_copy(st._h, -1))
    got = st.step(x)
    st.status()
    assert torch.equal(got, want)
    st.close()


def test_refusals():
    from kanjoos_b200.moe import FusedMoeStack
    banks, _ = _banks(803, 1, 16, 512, 256)
    with pytest.raises(Exception):
        FusedMoeStack(banks, top_k=4, n_tokens=65)     # more tokens than one launch takes
