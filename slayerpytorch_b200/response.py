"""Response and refractory kernels of the neuron models, as lists of samples.

Host arithmetic only: importing this module loads none of the operators."""
import math

import numpy as np


def alpha_kernel(tau, Ts, tSample, mult=1.0, epsilon=0.01):
    """Samples of mult * t/tau * exp(1 - t/tau) at t = 0, Ts, 2Ts, ..., cut where the tail
    drops below epsilon (src/slayer.py:114-123)."""
    taps = []
    for t in np.arange(0, tSample, Ts):
        value = mult * t / tau * math.exp(1 - t / tau)
        if abs(value) < epsilon and t > tau:
            break
        taps.append(value)
    return taps


def loihi_psp_kernel(neuron):
    """Impulse response of the Loihi current/voltage filter pair (src/slayerLoihi.py:66-79)."""
    keep_i = (1 << 12) - neuron['iDecay']
    keep_v = (1 << 12) - neuron['vDecay']
    u = 1 << (6 + neuron['wgtExp'] + 1)
    v = u
    out = [v]
    while v > 0:
        u = (u * keep_i) >> 12
        v = ((v * keep_v) >> 12) + u
        out.append(v)
    return [x / 2 for x in out]


def loihi_ref_kernel(neuron, scale=1000):
    """Refractory kernel equivalent of the Loihi reset (src/slayerLoihi.py:81-89)."""
    keep_v = (1 << 12) - neuron['vDecay']
    absolute = np.ones(neuron['refDelay']) * (-scale * neuron['theta'])
    absolute[0] = 0
    relative = [neuron['theta']]
    while relative[-1] > 0:
        relative.append((relative[-1] * keep_v) >> 12)
    return np.concatenate((absolute, -2 * np.array(relative))).astype('float32')
