// Device-side description of one render of a simulation (fp_sim_render): the camera, the
// render settings as the reference's RenderParams uniform holds them (volume-common.wgsl:4-10),
// the render box and the render pools.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fp_types.h"

#define FP_BLACKBODY_SIZE 512

// Depths a half-resolution pass records (VolumeSlices.ts DEPTH_SLICES).
#define FP_SLICES 8

// The render boxes' brick tables (FpRender::pages): rows of the box list, and the most bricks the
// boxes may hold together for the tables to be built (64 MB; a box is the span of a cluster's
// content, so thinly spread content can span far more bricks than it holds).
#define FP_BOX_INTS 8
#define FP_MAX_PAGES (1ll << 24)

struct FpRender {
  float ivp[16];  // clip to world, column-major
  int width, height;
  float time;
  float optical[4], light[4], smoke[4], fire[4];
  float sceneLight[3], ambient[3];
  float flameOpacity;
  int shadowSamples, raySteps, filter;
  int lightShift;       // lighting texels per brick side = 1 << lightShift
  const int* boxes;     // the render boxes, FP_BOX_INTS ints each: lo xyz, hi xyz in bricks
                        // (inclusive), the box's first entry in `pages`; boxes never overlap, each
                        // lies in one cluster of tiles
  int boxCount;
  int* pages;           // per box, x fastest, each brick's slot, -1 without one, or -2 - g for
                        // apron brick g; null when the boxes hold more than FP_MAX_PAGES bricks
                        // (lookups then go through the tile hash)
  long long pageCount;
  // Apron bricks: those without a slot that a brick with one precedes on some axes, so that a
  // sample based in that one reads them. The cells and texels such a sample can reach (those on
  // the brick's low faces) are computed once a render, per apron brick three planes (x = 0, then
  // y = 0, then z = 0, the axes left in x, y, z order). Past apronCap they are computed where a
  // sample needs them.
  int apronCap;
  int* apronCount;      // how many there are (it may exceed apronCap)
  int4* apronBricks;    // x, y, z, box
  float* apronField;    // the smoothed smoke of the field cells (no coarse smoke)
  float* apronSmoke;    // coarse smoke: the smoothed density of the coarse cells
  float4* apronLight;   // the incident light of the lighting texels
  float4* renderField;  // [slot][cell]: smoothed smoke, heat, lifetime, fuel (coarse smoke: the
                        // simulation's fields as they are)
  float2* units;        // [slot][block][4^3]: of each 2x2x2 cells of an 8^3 block, the most flame glow
                        // and the most smoke plus glow; null without room (taken from renderField then)
  float* renderSmoke;   // coarse smoke (smokeDiv > 1): [slot][smoke cells], the smoothed density
  float4* lighting;     // [slot][texel]: glow RGB, sun transmittance
  uint8_t* occupancy;   // [slot]: bit 0 flame glow, bit 1 anything visible, in the block and halo
  const float4* lut;    // blackbody: peak-normalised linear RGB, log2 radiance
  float* image;         // width x height x 4
  const float* depth;   // the scene's depth buffer (width x height, clip z 0..1), or null
  float4* slices;       // half resolution: FP_SLICES x sliceH x sliceW, or null (full resolution);
                        // without a scene depth only the last of them is read, and written
  int sliceW, sliceH;
};

// Launchers (fp_render.cu): the render pools of every active brick in the box, then the march.
void fp_launch_render(const SimParams* dP, const FpRender& R, int sms, cudaStream_t st);
// Scene-light sums (scene-lights.wgsl): 8 floats per anchor added into `sums` (zeroed).
void fp_launch_collect_lights(const SimParams* dP, const FpRender& R, const float* anchors, int count, float* sums,
                              int sms, cudaStream_t st);
// The blackbody table (blackbody.ts:85-97) computed on the host, FP_BLACKBODY_SIZE entries.
void fp_blackbody_table(float* out4);
