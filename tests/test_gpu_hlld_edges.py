"""HLLD faces whose inner (Alfven) wave stands exactly on the face while the star
state across it is unphysical: the reference computes both star states there
(SsL <= 0 and SsR >= 0, HLLD.cpp:66-100) and falls back to HLLE. The states were
found by a search on the CPU with the plain routine; the fast form has to take
the same way."""
import numpy as np
import pytest

from test_gpu_fast64 import lib, p, same_bits  # noqa: F401  (lib: the module's fixture)

pytestmark = pytest.mark.gpu

# rho p vx vy vz Bx By Bz of the left and the right state; the first half have
# SsL = 0 and an unphysical right star state, the others SsR = 0 and a left one
FACES = [
    ('0x1.3e69b0cb41781p+3 0x1.1274ac0307125p-4 0x1.0962568e4fa46p-1 0x1.7d421c538447ep+0 -0x1.5a0ac4ae12635p+0 -0x1.f3745e55ccf7bp+0 0x1.2ece196454aa2p+1 -0x1.74d0d9921194p-5',
     '0x1.437459a66f984p+0 0x1.3aa99d6baf3acp-3 -0x1.92ce5327919d1p+1 -0x1.9b3abc58d6048p-3 -0x1.445a415bf108fp+0 -0x1.f3745e55ccf7bp+0 -0x1.c5eaaa7fd6201p+1 -0x1.3b7dcdad68a2ap+1'),
    ('0x1.b11e84255f808p+0 0x1.9ab50c6b09f42p-7 0x1.6f8d605ab1594p-2 0x1.8e067d6a96708p-1 -0x1.480688e319362p+0 -0x1.7a44ae1818522p+0 -0x1.20a186a3b6bep-2 0x1.7ef88e4a7adc8p-1',
     '0x1.a8bad0dee606cp-1 0x1.3439d30ae130fp-10 0x1.6b16f1bc5e97ap-1 -0x1.15f63946305dcp-2 -0x1.9fda85c67d136p-1 -0x1.7a44ae1818522p+0 -0x1.a02b2abebbf1ep+1 -0x1.606abb225c768p+0'),
    ('0x1.51b41524bb769p+1 0x1.412227c90c03cp-4 0x1.5ee9002affca8p-2 0x1.d3aeb9b27a038p-2 -0x1.c37cb9f9441e7p+0 0x1.909baefe8f966p+0 -0x1.70e9f26e6aa44p-1 0x1.0227031096768p+1',
     '0x1.4c7254d18e5e1p-3 0x1.0b560872fbcep-3 -0x1.3eb8ff1b2040cp+0 -0x1.bedf58a0e391p+0 -0x1.42062ffa63ff6p+0 0x1.909baefe8f966p+0 0x1.5868abd40b3ap+1 0x1.730943cd5ae9p-1'),
    ('0x1.7b633ff1c138bp-3 0x1.504da052f4af7p-9 -0x1.26d3535c2fda9p-1 -0x1.ea789fea1b29p+0 -0x1.315c5468981ccp-1 -0x1.4d223a689f2fcp-2 0x1.a53b0b4ae64dap+1 -0x1.df32729ba90cp-3',
     '0x1.2085d19ddae86p-3 0x1.a3b1532b1bc0fp-5 0x1.4828e121ac81cp-3 -0x1.a46661cb18044p+0 0x1.cc37b0ce96c6p-3 -0x1.4d223a689f2fcp-2 0x1.289a86a102648p+1 -0x1.1d0c0fea062eap+1'),
    ('0x1.de004ec7de483p-1 0x1.0f3c4d3a5e591p-1 -0x1.4039394a846fep+0 0x1.4a79d162ec738p-2 -0x1.4710228fdac4p-5 -0x1.cec25e58a5017p+0 -0x1.29f1302683df9p+1 -0x1.2882bcef2be16p+1',
     '0x1.e13d0164504d9p-1 0x1.adc43e89d254fp-2 -0x1.39e4b350b0d2p-3 -0x1.d28daa6c19752p-1 -0x1.8580cceb39288p-3 -0x1.cec25e58a5017p+0 0x1.08de66cd297d8p-1 -0x1.25a4fb57e90bfp+1'),
    ('0x1.b60c7cae8aefdp-1 0x1.488fd50dced9dp-7 -0x1.8977a4312864ep-2 -0x1.0f2ff8eca443p-3 0x1.95ba6d2a1d218p+0 -0x1.28a50082c9a2ap-1 -0x1.a288eb3836d13p+1 -0x1.6c06ca884f2e2p+0',
     '0x1.49ea14954ed95p+0 0x1.cebb878abbf2dp-3 0x1.4fbca97b0d0d8p-4 0x1.89ccf14f711e8p-1 0x1.b4f47abdb68e8p-1 -0x1.28a50082c9a2ap-1 0x1.955bf14d4432p-2 0x1.8505738aadf26p+1'),
]


def test_standing_inner_wave(lib):
    L, R = (np.array([[float.fromhex(v) for v in f[k].split()] for f in FACES]) for k in (0, 1))
    out = np.zeros((2, len(FACES), 10))
    assert lib.f64_face(1, 3, len(FACES), p(L), p(R), 0.05, p(out)) == 0
    assert (out[1, :, 9] == 16).all()  # one HLLD to HLLE fallback in the plain routine
    assert same_bits(out[0], out[1]).all(), out
