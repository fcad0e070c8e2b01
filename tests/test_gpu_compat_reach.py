"""The compat render's noise march where its last sample lies beyond the far
point: with a step count barely above two the third sample is nearly two chords
from the near point, so coordinates that are moderate at both ends of the chord
are too large for the short floor there.

Reference: the same image with a second octave whose frequency takes the general
path for every sample.  Its weight of 1e-7 moves a sample's colour by at most
scale / 2 x 1e-7 and a pixel's, three samples over 1.05, by less than 1e-7."""
import numpy as np
import pytest

import cloudgb

pytestmark = pytest.mark.gpu

RADIUS = 2.0
REACH = 2.0e6  # scaled noise coordinate below which the short floor is taken


@pytest.mark.parametrize("share", [0.3, 0.75, 0.95, 0.999])
@pytest.mark.parametrize("eye", [(0.0, 0.0, -9.0), (9.0, 0.5, 1.0), (-6.0, 1.0, 6.0)])
def test_samples_beyond_the_far_point(ctx, eye, share):
    vol = cloudgb.CloudVolume(32, (-5.0, 5.0), (0.0, 0.0, 0.0), 4, ctx=ctx)
    vol.set_billboards(np.zeros((1, 3), np.float32), np.full(1, RADIUS, np.float32))
    vol.update()
    cam = cloudgb.Camera(eye, (0.0, 0.0, 0.0), width=64, height=48)
    # both ends of the middle chord at `share` of the reach
    adjust = RADIUS * 32.0 / (share * REACH)
    kw = dict(doConeTrace=False, adjustSize=adjust, stepSize=2.0 * RADIUS / adjust / 0.05,
              minNoiseSteps=2, maxNoiseSteps=3, noiseOpacity=-4.0)
    short = cloudgb.CompatShader(numOctaves=1, **kw).coneTrace(vol, cam)
    general = cloudgb.CompatShader(numOctaves=2, freqStep=1e7, persStep=1e-7,
                                   **kw).coneTrace(vol, cam)
    assert general[..., 0].std() > 0.02
    assert np.abs(short - general).max() <= 1e-6
