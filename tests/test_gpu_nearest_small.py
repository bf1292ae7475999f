"""Nearest facets on surfaces so small (coordinates around 2^-73) that squared distances lie in
the subnormal range of binary32, where the certified bounds by which leaves are culled lose
their digits: facets and closest points of pairs of facets almost equally far equal the
oracle's."""
import numpy as np
import pytest

import tetwild_gb300 as tw

pytestmark = pytest.mark.gpu


# point, then the six vertices of two facets; the second is nearer, by 0.2% to 6% in d^2
PAIRS = [
    "0x1.40240fad33237p-72 0x1.a2c14ece138e3p-71 -0x1.bb411c23929eap-71 "
    "-0x1.bbc1f8f124a46p-80 -0x1.b8d9562eb3052p-73 -0x1.808b73d75c95dp-72 "
    "0x1.8139d49077fedp-72 0x1.629885db8fef3p-71 -0x1.e8f8efe9f3ffdp-71 "
    "-0x1.541a2aa6bf93dp-74 -0x1.fd0f2eac663c1p-71 0x1.5e26861f45422p-72 "
    "0x1.4f5f3aa44646bp-72 0x1.2fcf74f8e334ep-71 -0x1.a36732db3a1a4p-71 "
    "0x1.791c3e235fb9dp-72 0x1.67483aa970743p-71 -0x1.5675bcbe04df1p-71 "
    "0x1.008f094be6981p-72 0x1.b7195da54a874p-71 -0x1.47764f3f6e419p-71",
    "-0x1.afb2c635e0b0dp-74 -0x1.1e146a3a75b9p-74 -0x1.902c407b7fd6dp-75 "
    "0x1.8f3e013804b03p-74 -0x1.472c776754bdcp-74 0x1.5c2ffa1226631p-75 "
    "-0x1.24980ad5195d4p-82 -0x1.940752f1a4342p-74 -0x1.06dd6cddf80d3p-74 "
    "-0x1.1b66ba79669a3p-78 -0x1.3defad6211394p-74 -0x1.d5a0e78d3bb7dp-75 "
    "0x1.358eaf250d1d9p-74 -0x1.97fffc5060ffap-76 0x1.6a524f356e6cdp-75 "
    "-0x1.27ec934b255c2p-74 -0x1.4f688d3b291c2p-74 0x1.db93948d19c7bp-75 "
    "-0x1.4caca31ac2e3ap-74 0x1.6c63f6a11f416p-74 -0x1.1e83ca05e6f78p-78",
    "0x1.a4540a0a4be55p-74 0x1.de6a9e46057d9p-74 0x1.1642564dbe776p-79 "
    "0x1.517cd33d1e6fp-77 -0x1.e0e49449d384bp-75 0x1.faf5b97f5fd0dp-77 "
    "-0x1.8bfc1e5992a84p-74 -0x1.d4aaf9cdd6865p-74 -0x1.6658e39da9f57p-75 "
    "0x1.f2621126150ccp-79 -0x1.896a767363f16p-76 -0x1.57660f919f943p-75 "
    "0x1.129c6353a8e29p-73 -0x1.fc0bd60cf6fccp-76 0x1.a0a2d6a89d21ap-73 "
    "0x1.6bc38cbc004cp-75 -0x1.7ea308e78b78fp-74 -0x1.942016c8d34a6p-73 "
    "0x1.68a95fc766fa4p-74 -0x1.eab14b8ef00dep-73 0x1.fe9dc1d50bae9p-73",
    "-0x1.aa6859b481393p-74 -0x1.9ce2e25cccf87p-74 0x1.d4941c6f3b9b8p-74 "
    "-0x1.be02c2fda583fp-80 0x1.4892ea140ed21p-74 -0x1.4aae20d5c10b6p-74 "
    "0x1.d308e4d78a445p-75 0x1.94100343f6e1p-74 0x1.88660c8e6602fp-75 "
    "-0x1.96190cbfa2bap-75 0x1.241f6106f2438p-77 0x1.0095ec324eb76p-75 "
    "0x1.9353c2e8401fep-73 0x1.b82bdd5d2987dp-74 -0x1.8963f3f2d7cbep-72 "
    "-0x1.dbc3f5f5a7d24p-74 0x1.da59adad33f16p-75 0x1.b5a186f2e6911p-74 "
    "-0x1.6f628f8ab823fp-74 -0x1.bc58e74497c6fp-75 -0x1.20b273ebdb542p-73",
    "-0x1.8837c2e9d86f5p-74 0x1.48caeccdccb2ep-75 0x1.d75b59535504dp-77 "
    "-0x1.b67268774e98dp-77 -0x1.16a59f1027d3ap-75 0x1.c1fafc836c9e8p-76 "
    "0x1.d9f55dd6681e6p-75 -0x1.95a44fb7b5016p-74 0x1.b240995f81ef8p-74 "
    "0x1.36767cef2563fp-74 -0x1.96d7d01c54131p-75 0x1.eb08efc5bb072p-75 "
    "-0x1.e4ba7e7ba68cp-77 0x1.0694da3c8e79p-75 -0x1.ef5ad576e7287p-75 "
    "0x1.4340ab877c739p-72 -0x1.44c88fbf0771p-79 0x1.512d051bc296ep-73 "
    "-0x1.e485102fe7cb4p-74 -0x1.6e29b3dce4fd2p-73 -0x1.57e4fdab76e55p-73",
    "-0x1.825b4490cd0a9p-75 0x1.9980194c10bd1p-74 -0x1.4c441722de69ap-75 "
    "0x1.4fbd0e3a89b75p-75 0x1.72f24b979e561p-74 -0x1.7f26bda5ac4a9p-74 "
    "-0x1.886d393741b91p-78 -0x1.2878b866b2c64p-79 0x1.0c726d0a12f39p-76 "
    "0x1.c5715a84fcebap-78 0x1.453329a964501p-74 -0x1.2151a0da5a56fp-74 "
    "-0x1.d32f725092cp-77 0x1.653b571c77eb5p-75 -0x1.b2f11ce750b14p-76 "
    "-0x1.1dc1af45e1fe7p-75 0x1.6edd66f1fae29p-75 -0x1.6b74d2ad23268p-77 "
    "-0x1.1aa31049d5447p-75 0x1.ba7395fda36bp-77 -0x1.8e1dbf8183ceep-77",
    "0x1.aef52fb667814p-81 0x1.f9992c3e27723p-76 -0x1.d5f4e4c4035a1p-75 "
    "0x1.5071571f8ee2fp-75 -0x1.af7ad7f8c3a8cp-74 0x1.2b8d65cfab841p-74 "
    "0x1.21fd51b466973p-76 0x1.36c50bdbe7e25p-76 -0x1.0b35cf555252ap-76 "
    "0x1.207146e12290dp-74 -0x1.b77ede2c7fdd1p-76 -0x1.147b9d987498ep-76 "
    "-0x1.1336d50855885p-75 -0x1.eb981605b343ep-77 -0x1.96248d06961b5p-75 "
    "0x1.7e42158166e15p-75 -0x1.68c268c2ad7b2p-77 -0x1.435037334ebd6p-75 "
    "-0x1.f36efc2e09451p-76 -0x1.8cd0560df582fp-74 0x1.8166869e15674p-74",
]


@pytest.mark.parametrize("pair", PAIRS, ids=range(len(PAIRS)))
def test_nearest_on_a_tiny_surface(ctx, oracle, pair):
    x = np.array([float.fromhex(h) for h in pair.split()]).reshape(7, 3)
    V, F, P = x[1:], np.array([[0, 1, 2], [3, 4, 5]], np.int32), x[:1]
    eps = 1e-20
    ctx.set_params(eps * eps, eps)
    ctx.surface_upload(V, F)
    wq, wd, wf = oracle.surface(V, F).nearest(P)
    assert wf[0] == 1 and wd[0] <= eps * eps
    for prec in (tw.TW_PRECISION_FP64, tw.TW_PRECISION_FP32_CERTIFIED):
        ctx.set_precision(prec)
        try:
            q, d, f = ctx.nearest_points(P)
        finally:
            ctx.set_precision(tw.TW_PRECISION_FP64)
        assert np.array_equal(f, wf) and np.array_equal(d, wd) and np.array_equal(q, wq)
