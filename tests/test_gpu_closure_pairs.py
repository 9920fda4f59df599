"""The learned closure's step on both spheres of a pair: a network with a known
constant output gives every bridge a force that plain numpy can state; and the
contact angles its steps run with."""
import copy

import numpy as np
import pytest

import _workloads
from gpucode_gb300 import _abi, configs
from gpucode_gb300.capnet import CapNet
from gpucode_gb300.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("output", [1.0, 0.7])
def test_constant_network_pulls_both_spheres_alike(cuda, output):
    """Wet minus dry forces of one step from rest are the bridges' alone:
    -2 pi R_eff gamma output along the pair's normal on one sphere, the opposite
    on the other.  1.0 is a value like any other.  A network without last-layer
    weights returns y_mean exactly; the two runs' sums (FP32, compensated) round
    once each, the normals and products a few times: 2e-6 of the largest sum."""
    w = _workloads.small_wet()
    w.inp.cut_gap = 1.5
    dry = copy.deepcopy(w.inp)
    dry.force_cap = 0
    setups = {"wet": configs.Setup.build(w.inp, w.dia), "dry": configs.Setup.build(dry, w.dia)}
    for setup in setups.values():  # a thick film: six bridges a sphere
        setup.s.lqd.layer = 0.3
        setup.s.prm.SearchGap = 0.38
    p = np.zeros(4610, np.float32)
    norm = np.array([0] * 4 + [1] * 4 + [output, 2.0] + [1] * 2 + [-1e3] * 4 + [1e3] * 4, np.float32)
    net = CapNet(seed=0)
    net.set(p, norm)
    pos = w.pos0_reduced
    force = {}
    for name, cap in (("wet", "mlp"), ("dry", "formula")):
        e = Engine(setups[name], precision="mixed", capillary=cap)
        if cap == "mlp":
            e.set_capnet(net)
        e.set_state(pos)
        e.step(1)
        e.sync()
        force[name] = e.get_state()["force"]
        if name == "wet":
            n, partners = e.neighbors()
            _, brg = e.history(int(n.max()))
            assert e.stats()["cap_mlp"] > 0 and e.stats()["cap_fallback"] == 0
        e.close()
    net.close()
    rad, gamma = w.setup.rad, w.setup.s.lqd.stension
    want = np.zeros_like(pos)
    bridges = 0
    for i in range(len(n)):
        for a in np.flatnonzero(brg[i, : n[i]] == 1):
            j = int(partners[i, a])
            d = pos[i] - pos[j]
            effr = 2 * rad[i] * rad[j] / (rad[i] + rad[j])
            want[i] -= 2 * np.pi * effr * gamma * output * d / np.linalg.norm(d)
            bridges += 1
    assert bridges > 96 * len(n) / 32  # a warp of spheres queues more than it holds at once
    scale = max(np.abs(f).max() for f in force.values())
    assert np.abs(force["wet"] - force["dry"] - want).max() <= 2e-6 * scale


@pytest.mark.parametrize("first", [1, 3])
def test_contact_angles_set_between_steps_are_used(cuda, first):
    """Steps chained on the device after the angles were changed give the bits
    of host-driven steps, which read the angles at every launch; and a liquid
    model is still refused after the first step"""
    w = _workloads.small_wet()
    pos, vel, ang = _workloads.stirred(w, vscale=0.05, wscale=0.1)
    rng = np.random.default_rng(3)
    norm = np.array([-6, -6, 0.3, 0.6] + [2, 2, 0.1, 0.2] + [0.8, 0.1] + [0.2, 0.02] + [-1e3] * 4 + [1e3] * 4,
                    np.float32)
    net = CapNet(seed=0)
    net.set((0.3 * rng.standard_normal(4610)).astype(np.float32), norm)
    out = []
    for graph, change in ((True, True), (False, True), (True, False)):
        e = Engine(w.setup, precision="mixed", capillary="mlp", use_graph=graph)
        e.set_capnet(net)
        e.set_state(pos, vel, ang)
        e.step(first)
        if change:
            e.set_contact_angles(0.9, seed=11)
        if graph:
            with pytest.raises(_abi.DemError):
                e.set_liquid_model("per_contact", seed=2)
        e.step(3)
        e.step(1)
        e.sync()
        out.append(e.get_state())
        e.close()
    net.close()
    for k in ("pos", "vel", "angvel", "force"):
        np.testing.assert_array_equal(out[0][k], out[1][k])
    assert np.abs(out[0]["force"] - out[2]["force"]).max() > 0
