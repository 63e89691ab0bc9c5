"""The work that users of this package have it do, as cases that can be timed and compared.

A case is one call of the public layer interface on tensors of a stated shape ``[N, C, H, W, T]``:

``delay``    ``delay(spike(psp(x)))`` of a spiking dense layer and its backward; ``x`` is the weighted input of the
             layer.  ``learn``: the delays are a parameter; ``fused``: through ``spikeDelayed``.
``deep``     ``psp(spike(psp(x)))`` and its backward: a layer whose spikes go on to the next layer's filter.
             ``fused``: through ``spikePsp``, the spikes staying bit-packed.
``input``    ``psp`` of a spike tensor, no gradient: the filter in front of a network's first layer.
``infer``    ``spike(psp(x))`` without gradients.
``loss``     psp, spike, the spike-count loss and its gradient: the last layer of a training step.
``loihi``    ``delayShift(spikeLoihi(w), 1)`` and its backward, or (``grad`` false) forward only.
             ``fused``: through ``spikeLoihiDelayed``.
``events``   a recording's address events, host arrays as a file reader returns them, to a spike tensor.
"""
import math

import numpy as np
import torch

from slayerpytorch_b200.layer import loihiLayer, spikeLayer
from slayerpytorch_b200.loss import spikeClassifier, spikeLoss
from slayerpytorch_b200.spikeio import event


def listed():
    return [
        # one dense layer of 512 neurons, four samples: an experiment's first network, bound by latency
        _case("dense_chain", "delay", (4, 512, 1, 1, 300), learn=False, fused=False),
        # the hidden layer of the 2312-512-10 classifier at its training batch, delays learned
        _case("mlp_hidden", "delay", (64, 512, 1, 1, 300), learn=True, fused=False),
        # the output layer of that classifier with the loss of its training step
        _case("mlp_output_loss", "loss", (64, 10, 1, 1, 300)),
        # one recording of a 34 x 34 sensor made into the network's input, once per sample by a data loader
        _case("events_34x34", "events", (1, 2, 34, 34, 300), count=5000),
        # the filter in front of the CNN's first layer, on a batch of 34 x 34 frames with 5 % spikes
        _case("cnn_input_psp", "input", (128, 2, 34, 34, 300), rate=0.05),
        # the CNN's first hidden layer at its training batch: the largest of the SRM networks
        _case("cnn_first", "deep", (128, 16, 32, 32, 300), fused=True),
        # a deeper layer of the CNN through the methods a network written for the reference calls
        _case("cnn_third", "deep", (128, 64, 8, 8, 300), fused=False),
        # a small evaluation batch of the CNN, an odd number of neurons' rows and of time steps
        _case("cnn_infer_odd", "infer", (11, 16, 33, 33, 301)),
        # both layers of the 200-256-200 network are about this size: long sequences, learned delays
        _case("long_sequence", "delay", (32, 256, 1, 1, 2000), learn=True, fused=True),
        # the hidden layer of a small Loihi classifier, T = 350, batch 12
        _case("loihi_mlp", "loihi", (12, 512, 1, 1, 350), fused=False, grad=True),
        # the first layer of the Loihi gesture CNN at its training batch: the largest work of all
        _case("loihi_first", "loihi", (64, 16, 32, 32, 1450), fused=True, grad=True),
        # a deeper layer of the Loihi CNN when it is evaluated
        _case("loihi_infer", "loihi", (64, 32, 8, 8, 1450), fused=False, grad=False),
    ]


def _case(name, kind, shape, **options):
    case = {"kind": kind, **dict(zip("NCHWT", shape)), "tauSr": 10.0, **options}
    if name:
        case["name"] = name
    return case


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["delay", "delay", "deep", "deep", "input", "infer", "loss", "loihi", "loihi", "events"])
    tau = rng.choice([5.0, 10.0, 10.0, 10.0])
    N, flag = log(4, 128), rng.random() < 0.5
    if kind == "events":
        side = rng.choice([34, 34, 64, 128])
        return _case(None, kind, (1, 2, side, side, log(200, 1450)), count=log(1000, 300000))
    if kind == "loss":
        return _case(None, kind, (N, rng.randint(2, 25), 1, 1, log(100, 2000)))
    if kind == "delay":
        case = _case(None, kind, (N, log(64, 1024), 1, 1, log(150, 2000)), learn=rng.random() < 0.7, fused=flag)
    elif kind == "input":
        side = rng.randint(16, 64)
        case = _case(None, kind, (N, rng.randint(1, 2), side, side, log(150, 1450)), rate=rng.choice([0.01, 0.02, 0.05, 0.1]))
    else:
        side = rng.randint(4, 34)
        case = _case(None, kind, (N, rng.choice([8, 16, 32, 64]), side, side, log(150, 1450)))
        if kind == "deep":
            case["fused"] = flag
        if kind == "loihi":
            case.update(fused=flag, grad=rng.random() < 0.7)
    case["tauSr"] = tau
    while _size(case) > 400_000_000:
        case["N"] = (case["N"] + 1) // 2
    return case


def _size(case):
    return case["N"] * case["C"] * case["H"] * case["W"] * case["T"]


def _srm(case, Ts=1.0):
    neuron = {"type": "SRMALPHA", "theta": 10, "tauSr": case["tauSr"], "tauRef": 1.0, "scaleRef": 2, "tauRho": 1, "scaleRho": 1}
    return neuron, {"Ts": Ts, "tSample": case["T"]}


def _loihi(case):
    neuron = {"type": "LOIHI", "vThMant": 80, "vDecay": 128, "iDecay": 1024, "refDelay": 1, "wgtExp": 0, "tauRho": 1, "scaleRho": 1}
    return neuron, {"Ts": 1, "tSample": case["T"]}


def prepare(case, seed):
    kind = case["kind"]
    shape = tuple(case[k] for k in "NCHWT")
    if kind == "events":
        rng = np.random.default_rng(seed)
        n, T = case["count"], case["T"]
        return {"kind": kind, "shape": shape[1:], "x": rng.integers(0, case["W"], n), "y": rng.integers(0, case["H"], n),
                "p": rng.integers(0, 2, n), "t": np.sort(rng.uniform(0.0, 1.02 * T, n))}    # the last events fall off the end
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    normal = lambda: torch.empty(shape, device=dev).normal_(generator=gen)
    state = {"kind": kind, "case": dict(case)}
    if kind == "loihi":
        state["net"] = loihiLayer(*_loihi(case)).to(dev)
        # integer weights over sparse input spikes: one in ten samples gets a weighted spike
        w = torch.randint(-128, 128, shape, device=dev, generator=gen, dtype=torch.int16).float()
        for part in w:
            part.mul_(torch.rand(part.shape, device=dev, generator=gen) < 0.1)
        if case["grad"]:
            state["g"] = normal()
            w.requires_grad_(True)
        state["x"] = w
        return state
    neuron, simulation = _srm(case)
    state["net"] = spikeLayer(neuron, simulation).to(dev)
    if kind == "input":
        x = torch.rand(shape, device=dev, generator=gen)
        state["x"] = x.lt_(case["rate"])
        return state
    # weighted input whose filtered potential has a standard deviation of 0.55 theta: a few percent of spikes
    x = normal().mul_(5.5 / (math.e * math.sqrt(case["tauSr"] / 4)))
    if kind == "loss":
        start, stop = 0, case["T"]
        error = {"type": "NumSpikes", "tgtSpikeRegion": {"start": start, "stop": stop}, "tgtSpikeCount": {True: 60, False: 10}}
        state["loss"] = spikeLoss({"neuron": neuron, "simulation": simulation, "training": {"error": error}}).to(dev)
        label = torch.randint(0, case["C"], (case["N"],), device=dev, generator=gen)
        state["desired"] = torch.nn.functional.one_hot(label, case["C"]).float().reshape(shape[:4] + (1,))
    if kind == "delay":
        most = 5.0 if case["T"] < 1000 else 10.0
        delays = torch.rand((case["C"], case["H"], case["W"]), device=dev, generator=gen) * most
        if case["learn"]:
            state["delay"] = state["net"].delay((case["C"], case["H"], case["W"])).to(dev)
            state["delay"].delay.data.copy_(delays)
        else:
            state["delay"] = delays
    if kind in ("delay", "deep"):
        state["g"] = normal()
    state["x"] = x.requires_grad_(kind != "infer")
    return state


def run(state):
    kind = state["kind"]
    if kind == "events":
        spikes = torch.zeros(state["shape"], device="cuda")
        return event(state["x"], state["y"], state["p"], state["t"]).toSpikeTensor(spikes)
    case, net, x = state["case"], state["net"], state["x"]
    if kind == "input":
        with torch.no_grad():
            return net.psp(x)
    if kind == "infer":
        with torch.no_grad():
            return net.spike(net.psp(x))
    if kind == "loihi":
        if not case["grad"]:
            with torch.no_grad():
                return _loihi_forward(case, net, x)
        out = _loihi_forward(case, net, x)
        return [out, *torch.autograd.grad(out, [x], state["g"])]
    if kind == "loss":
        spikes = net.spike(net.psp(x))
        loss = state["loss"].numSpikes(spikes, state["desired"])
        (grad,) = torch.autograd.grad(loss, [x])
        return [spikes.detach(), loss.detach(), grad, spikeClassifier.getClass(spikes.detach(), host=False)]
    if kind == "deep":
        u = net.psp(x)
        if case["fused"]:
            out, packed = net.spikePsp(u)
            return [out.detach(), packed.bits, *torch.autograd.grad(out, [x], state["g"])]
        spikes = net.spike(u)
        out = net.psp(spikes)
        return [out.detach(), spikes.detach(), *torch.autograd.grad(out, [x], state["g"])]
    delay = state["delay"]
    wanted = [x, delay.delay] if case["learn"] else [x]
    u = net.psp(x)
    if case["fused"]:
        out = net.spikeDelayed(u, delay)
    elif case["learn"]:
        out = delay(net.spike(u))
    else:
        out = net.delayShift(net.spike(u), delay)
    return [out.detach(), *torch.autograd.grad(out, wanted, state["g"])]


def _loihi_forward(case, net, w):
    return net.spikeLoihiDelayed(w, 1) if case["fused"] else net.delayShift(net.spikeLoihi(w), 1)


def work(case):
    n, kind = _size(case), case["kind"]
    # taps of the filter: where t/tau exp(1 - t/tau) falls below a hundredth; 110 for the Loihi response
    taps = 110 if kind == "loihi" else min(case["T"], 7.64 * case["tauSr"])
    if kind == "events":
        return {"bytes": 4 * n + 32 * case["count"], "flops": 0}                # 32: four 8-byte host arrays
    if kind in ("input", "infer"):
        return {"bytes": 8 * n, "flops": 2 * taps * n}
    if kind == "loihi":
        return {"bytes": 16 * n, "flops": (2 * taps + 24) * n} if case["grad"] else {"bytes": 8 * n, "flops": 12 * n}
    if kind == "loss":
        return {"bytes": 12 * n, "flops": 8 * taps * n}
    # weighted input and gradient in, result and gradient out; deep: the spikes too, and both filters
    if kind == "deep":
        return {"bytes": (16.125 if case["fused"] else 20) * n, "flops": 8 * taps * n}
    return {"bytes": 16 * n, "flops": 4 * taps * n}


def tolerance(case):
    # 32-bit sums of some hundred terms; spikes, their positions and the binned events are exact beside them
    return {"rel": 1e-5}
