// afx_stream.cu -- the rigid multi-camera reconstruction stream (af::startMeshReconstructionStream,
// src/MeshRecontructionStream.cu:115-206), device-resident.
//
// Per frame, for every camera (CameraData::processNextFrame, :88-112): depth from uint16 mm,
// runFilterDepthKernel, the bilateral filter when enabled, and DeviceDepthImage::backProject
// (include/af/DeviceImage.cuh:54-58): runDepthToMeshKernel with the camera's intrinsics, then
// runTransformKernel with the inverse of its world-to-camera transform.  The cameras' clouds are
// concatenated in camera order (every pixel, invalid ones included).  The volume is re-initialised
// (DeviceTsdf::initDefault) and -- as the reference does -- only camera 0's filtered depth is
// integrated, at the volume's centre and rotation (DeviceTsdf::integrate ->
// runIntegrateTSDFFromFrameKernel), and the full marching-cubes mesh is extracted (untranslated).
// Nothing is read back to the host; the outputs are device views.
#include <cstring>
#include <new>

#include "afx_internal.h"

using namespace afx;

struct afx_rigid_stream {
    afx_rigid_stream_params p;
    Volume vol;
    long S = 0, P = 0;
    void* arena = nullptr;
    float* depth;    // [n_cameras * P], the filtered depth of each camera
    float* cloud;    // [n_cameras * P * 3]
    float* tsdf;
    float* weights;
    float* verts;    // [3 * triangle_capacity * 3]
    int* faces;      // [triangle_capacity * 3]
    unsigned* counts;  // faces, vertices
    int* error;
    unsigned char* occ;   // per 8^3 brick of the volume: 1 where this frame left a positive value
    unsigned* mc_tiles;   // marching cubes: count + occupied tiles
    uint32_t* umap;    // [n_cameras * P * 2], undistortion maps of the distorted cameras
};

extern "C" {

void afx_rigid_stream_default_params(afx_rigid_stream_params* p) {
    if (!p) return;
    std::memset(p, 0, sizeof(*p));
    p->n_cameras = 1;
    p->width = 640;
    p->height = 576;
    for (int c = 0; c < AFX_MAX_CAMERAS; ++c) {
        const float K[9] = {504.f, 0.f, 0.f, 0.f, 504.f, 0.f, 320.f, 288.f, 1.f};
        std::memcpy(p->K[c], K, sizeof(K));
        for (int i = 0; i < 16; ++i) p->camera_to_world[c][i] = (i % 5 == 0) ? 1.f : 0.f;
    }
    p->dims[0] = p->dims[1] = p->dims[2] = 400;  // Settings.cpp: tsdfDim
    p->volume_size[0] = p->volume_size[1] = p->volume_size[2] = 1.f;  // tsdfSize
    p->delta = 0.016f;
    for (int i = 0; i < 9; ++i) p->rotation[i] = (i % 4 == 0) ? 1.f : 0.f;
    p->depth_threshold = 1.2f;
    p->bilateral = 1;
    p->bilateral_r = 2;
    p->sigma_i = 0.03f;
    p->sigma_s = 2.f;
    p->bilateral_thr = 0.09f;
    p->triangle_capacity = 4000000;
}

int afx_rigid_stream_create(const afx_rigid_stream_params* params, afx_rigid_stream** out) {
    if (!params || !out) return AFX_ERR_INVALID_ARGUMENT;
    const afx_rigid_stream_params& p = *params;
    if (p.n_cameras < 1 || p.n_cameras > AFX_MAX_CAMERAS || p.width < 3 || p.height < 3 || p.dims[0] < 3 ||
        p.dims[1] < 3 || p.dims[2] < 3 || p.triangle_capacity < 1 || (p.bilateral && p.bilateral_r < 1))
        return AFX_ERR_INVALID_ARGUMENT;
    afx_rigid_stream* s = new (std::nothrow) afx_rigid_stream();
    if (!s) return AFX_ERR_NO_MEMORY;
    s->p = p;
    float vs[3];
    for (int c = 0; c < 3; ++c) vs[c] = p.volume_size[c] / (float)p.dims[c];  // DeviceTsdf::voxelSize
    s->vol = make_volume(p.dims, vs, p.volume_size);
    s->S = (long)p.dims[0] * p.dims[1] * p.dims[2];
    s->P = (long)p.width * p.height;
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t nc = (size_t)p.n_cameras, P = (size_t)s->P, S = (size_t)s->S, T = (size_t)p.triangle_capacity;
    bool distorted = false;
    for (int c = 0; c < p.n_cameras; ++c) distorted = distorted || p.distortion[c].is_distorted;
    const size_t bricks = (size_t)((p.dims[0] + 7) / 8) * ((p.dims[1] + 7) / 8) * ((p.dims[2] + 7) / 8);
    const size_t sizes[] = {nc * P * 4, nc * P * 12, S * 4, S * 4, T * 36, T * 12, 64, 64,
                            bricks, mc_tile_ws_words(s->vol) * 4, distorted ? nc * P * 8 : 0};
    constexpr int kBuffers = (int)(sizeof(sizes) / sizeof(sizes[0]));
    size_t total = 0;
    for (size_t x : sizes) total += al(x);
    cudaError_t e = cudaMalloc(&s->arena, total);
    if (e != cudaSuccess) {
        note_cuda_error(e);
        delete s;
        return AFX_ERR_NO_MEMORY;
    }
    char* q = static_cast<char*>(s->arena);
    void* ptr[kBuffers];
    for (int i = 0; i < kBuffers; ++i) {
        ptr[i] = q;
        q += al(sizes[i]);
    }
    s->depth = (float*)ptr[0];
    s->cloud = (float*)ptr[1];
    s->tsdf = (float*)ptr[2];
    s->weights = (float*)ptr[3];
    s->verts = (float*)ptr[4];
    s->faces = (int*)ptr[5];
    s->counts = (unsigned*)ptr[6];
    s->error = (int*)ptr[7];
    s->occ = (unsigned char*)ptr[8];
    s->mc_tiles = (unsigned*)ptr[9];
    s->umap = distorted ? (uint32_t*)ptr[10] : nullptr;
    e = cudaMemset(s->arena, 0, total);
    // each distorted camera's cv::initUndistortRectifyMap(CV_32FC1) map, built once
    // (src/MeshRecontructionStream.cu:97-98 rebuilds the same map every frame)
    int map_rc = AFX_OK;
    for (int c = 0; c < p.n_cameras && e == cudaSuccess && !map_rc; ++c)
        if (p.distortion[c].is_distorted)
            map_rc = undistort_map_impl(s->umap + (size_t)c * P * 2, p.width, p.height, p.K[c], &p.distortion[c],
                                        AFX_UNDISTORT_NEAREST, nullptr);
    if (e == cudaSuccess && !map_rc) e = cudaStreamSynchronize(nullptr);
    if (map_rc) {
        cudaFree(s->arena);
        delete s;
        return map_rc;
    }
    if (e != cudaSuccess) {
        cudaFree(s->arena);
        delete s;
        return note_cuda_error(e);
    }
    *out = s;
    return AFX_OK;
}

int afx_rigid_stream_destroy(afx_rigid_stream* s) {
    if (!s) return AFX_ERR_INVALID_ARGUMENT;
    cudaDeviceSynchronize();
    const cudaError_t e = cudaFree(s->arena);
    delete s;
    return note_cuda_error(e);
}

int afx_rigid_stream_process(afx_rigid_stream* s, const uint16_t* const* depth_mm, void* stream) {
    if (!s || !depth_mm) return AFX_ERR_INVALID_ARGUMENT;
    const afx_rigid_stream_params& p = s->p;
    for (int c = 0; c < p.n_cameras; ++c)
        if (!depth_mm[c]) return AFX_ERR_INVALID_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    const long P = s->P;
    StreamPrep A;
    A.width = p.width;
    A.height = p.height;
    A.depth_threshold = p.depth_threshold;
    A.bilateral = p.bilateral;
    for (int c = 0; c < p.n_cameras; ++c) {
        StreamCamera& cam = A.cam[c];
        cam.mm = depth_mm[c];
        // a distorted camera's filtered frame is overwritten by the undistortion of the unfiltered metres
        // (src/MeshRecontructionStream.cu:91-101)
        cam.umap = p.distortion[c].is_distorted ? s->umap + (size_t)c * P * 2 : nullptr;
        cam.depth = s->depth + c * P;
        cam.cloud = s->cloud + 3 * c * P;
        cam.K = make_intrinsics(p.K[c]);
        cam.fxi = 1.0f / p.K[c][0];
        cam.fyi = 1.0f / p.K[c][4];
        std::memcpy(cam.T, p.camera_to_world[c], sizeof(cam.T));
    }
    int rc = stream_prep_impl(A, p.n_cameras, p.bilateral_r, p.sigma_i, p.sigma_s, p.bilateral_thr, st);
    if (rc) return rc;
    // DeviceTsdf::initDefault + integrate(cameras[0]) in one write-only pass, which also says which bricks
    // marching cubes has to look at
    AFX_CUDA(cudaMemsetAsync(s->counts, 0, 8, st));
    rc = integrate_fresh_impl(s->tsdf, s->weights, s->depth, p.width, p.height, p.delta, s->vol, p.rotation,
                              p.center, p.K[0], st, s->occ);
    if (rc) return rc;
    const long T = p.triangle_capacity;
    rc = mc_fused_impl(s->tsdf, s->weights, kVoxF32, s->vol, 0.f, nullptr, nullptr, 0, s->verts, s->counts + 1, T * 3,
                       s->faces, s->counts, T, st, s->error, kMcTilePipe4, s->occ, s->mc_tiles, true);
    return rc;
}

int afx_rigid_stream_outputs(afx_rigid_stream* s, float** cloud, long* cloud_points, float** vertices,
                             unsigned** vertex_count, int** faces, unsigned** face_count, float** tsdf, float** weights) {
    if (!s) return AFX_ERR_INVALID_ARGUMENT;
    if (cloud) *cloud = s->cloud;
    if (cloud_points) *cloud_points = s->P * s->p.n_cameras;
    if (vertices) *vertices = s->verts;
    if (vertex_count) *vertex_count = s->counts + 1;
    if (faces) *faces = s->faces;
    if (face_count) *face_count = s->counts;
    if (tsdf) *tsdf = s->tsdf;
    if (weights) *weights = s->weights;
    return AFX_OK;
}

}  // extern "C"
